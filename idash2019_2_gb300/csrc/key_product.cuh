// Negacyclic product of TRLWE masks with a binary key on the tensor cores
// (key_product.cu), for decryption and encryption.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace idash {

constexpr uint32_t kKeyMaxN = 2048;

// A binary key, by value in the launch parameters: bit i % 32 of word i / 32
// is coefficient i.
struct KeyBits {
    uint32_t w[kKeyMaxN / 32];
};

// Whether `key` has only the coefficients 0 and 1; its bits into *out.
bool key_bits(const int32_t *key, uint32_t N, KeyBits *out);

// N the product kernel is built for (a power of two).
inline bool key_product_supported(uint32_t N) { return N >= 32 && N <= kKeyMaxN; }

struct KeyProductArgs {
    KeyBits key;
    uint8_t *rows;            // coefficient 0 of row 0: the mask a[0..N), then the body b[0..N)
    uint64_t stride;          // bytes, a multiple of 4
    const uint32_t *row_map;  // row r is at row_map[r] (null: r)
    uint64_t n_rows;
    uint32_t N, n_coef;       // coefficients wanted: [0, n_coef)
    float *scores;            // see launch_key_product
    uint32_t *err;            // device error word
    // set by the launch
    uint32_t tile_cols, pairs, vec_rows, vec_scores;
    uint64_t items;
};

// scores non-null: scores[r * n_coef + j] = float((b - a*s)[j] / 2^32).
// scores null: b[j] += (a*s)[j] in place.  Bodies that the product does not get
// into (the launch fails, or a wait on the device expires) are cleared: they
// hold messages.
cudaError_t launch_key_product(KeyProductArgs a, int sm_count, cudaStream_t s);

// Allows the kernels their shared memory (once per device, before any launch or capture).
cudaError_t configure_key_product();

}  // namespace idash
