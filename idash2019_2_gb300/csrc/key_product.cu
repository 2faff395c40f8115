// a*s mod (X^N + 1, 2^32) for many masks a and one binary key s (tLwePhase and
// tLweSymEncryptZero, eval/idash.cpp:714 and :625) as a matrix product on
// tcgen05.mma:  P[row][j] = sum_k a[row][k] T[k][j],  T[k][j] = s[j - k] for
// j >= k and -s[N + j - k] below.
//
// Exactness.  A mask word is three unsigned digits, x = u0 + 2^11 u1 +
// 2^22 u2 (11, 11 and 10 bits).  The fp16 bit patterns 0 .. 0x7FF are the
// values u * 2^-24 (the subnormals and the first binade are one linear
// scale), so a digit is its own encoding: no conversion instruction.  T holds
// 0, 1 and -1.  A digit's sum over k stays below N * 2047 < 2^22 units of
// 2^-24, which fp32 holds exactly; adding 0.75 (whose last place is 2^-24)
// makes its bits an integer, and P = sum_i 2^(11 i) D_i mod 2^32.
//
// Layout.  M = 128 of an MMA is 40 rows x 3 digits (quadrant w of the TMEM
// lanes: digit d of row 10 w + r in lane 32 w + 10 d + r), N = up to 256
// coefficients j.  T is Toeplitz and an 8 x 8 core matrix of it depends only
// on the difference of its group indices, so with the k-groups in reverse
// order the whole of T is a table of 2N/8 - 1 core matrices (32 KB at
// N = 1024) that the descriptor walks with both strides 128 bytes: it is
// built once per CTA from the key bits and never reloaded.
//
// Structure: one CTA of 14 warps per SM, persistent over items (40 rows, a
// pair of column tiles t0, t1).
//   warps 9-13 load 64-word pieces of the rows (two pieces ahead, in
//              registers), split them into digits, store them as the MMA's A
//              (k-groups 16 bytes off a multiple of 128 apart, so that the
//              eight groups of a row, one per lane, are in different banks);
//   warp 8     issues the MMAs: t0 over chunk g and t1 over chunk g - kLag, so that one tile's epilogue runs under the other's
//              MMAs although the two accumulators (2 x 256 columns) fill TMEM;
//   warps 0-3  epilogue of t0, warps 4-7 of t1: each lane turns its digit sums
//              into shifted words, three lanes exchange them (two shuffles per
//              three words), and every lane finishes 4 consecutive
//              coefficients of a row out of 12.
// Every wait is bounded and ends when another role raised the abort flag.
//
// What bounds it: 242,646 masks x 1,000 coefficients take 1.67 ms (7.00 ms as
// sums over the key's set bits on CUDA cores).  The MMAs alone would take 0.7
// ms and reading and writing 3.0 GB 0.45 ms; one item (40 rows x 512
// coefficients) takes 41,000 cycles, of which the MMAs' operands keep shared
// memory busy for 12,300 and the MMA warp waits 15,000 for an epilogue, whose
// shuffles and 16-byte accesses share the same pipe.
#include <algorithm>

#include "key_product.cuh"
#include "tcgen05.cuh"

namespace idash {

bool key_bits(const int32_t *key, uint32_t N, KeyBits *out) {
    *out = KeyBits{};
    for (uint32_t i = 0; i < N; ++i) {
        if (key[i] != 0 && key[i] != 1) return false;
        out->w[i / 32] |= uint32_t(key[i]) << (i % 32);
    }
    return true;
}

namespace {

constexpr uint32_t kRows = 40;        // rows per item
constexpr uint32_t kChunkWords = 64;  // mask words per pipeline chunk (four K = 16 steps)
constexpr uint32_t kStages = 8;       // chunks of A in shared memory
constexpr uint32_t kLag = 4;          // t1 runs this many chunks behind t0
constexpr uint32_t kGroupBytes = 128 * 16 + 16;  // one k-group (8 words) of A: 16 core matrices and the padding
constexpr uint32_t kStageBytes = (kChunkWords / 8) * kGroupBytes;
constexpr uint32_t kTileMax = 256;    // columns of one accumulator
constexpr uint32_t kMmaWarp = 8, kConvWarp0 = 9, kConvWarps = 5;
constexpr uint32_t kKpThreads = 32 * (kConvWarp0 + kConvWarps);
constexpr uint32_t kHeader = 1024;
constexpr uint32_t kMagicBits = 0x3F400000u;  // 0.75f
static_assert(kLag < kStages, "t1's chunks must still be in the ring");
static_assert(kRows * (kChunkWords / 8) == 2 * 32 * kConvWarps, "two 8-word units per converter thread and chunk");

struct KpShared {
    uint64_t a_full[kStages], a_empty[kStages];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t drain;
    uint32_t tmem_base, abort;
    uint32_t key[kKeyMaxN / 32];
};
static_assert(sizeof(KpShared) <= kHeader, "header area");

__host__ __device__ constexpr uint32_t kp_table_bytes(uint32_t N) { return (2 * N / 8) * 128; }
// at least 120 KB, so that no second CTA (which would wait for this one's
// tensor memory) fits on the SM
constexpr size_t kp_smem(uint32_t N) { return kHeader + kp_table_bytes(N) + size_t(kStages) * kStageBytes; }
static_assert(kp_smem(64) > 120 * 1024, "one CTA per SM");

__device__ __forceinline__ const uint8_t *kp_row(const KeyProductArgs &a, uint64_t r) {
    return a.rows + (a.row_map ? uint64_t(a.row_map[r]) : r) * a.stride;
}

// 4 (n = 1) or 8 (n = 2) words from p: 16-byte loads when the rows allow them.
template <int kVecs>
__device__ __forceinline__ void kp_load(const uint32_t *p, bool vec, uint32_t (&v)[4 * kVecs]) {
    if (vec) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            const uint4 q = reinterpret_cast<const uint4 *>(p)[i];
            v[4 * i] = q.x;
            v[4 * i + 1] = q.y;
            v[4 * i + 2] = q.z;
            v[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4 * kVecs; ++i) v[i] = p[i];
    }
}

// T's entry at difference d = j - k as fp16 bits.
__device__ __forceinline__ uint32_t kp_entry(const uint32_t *key, uint32_t N, int32_t d) {
    const uint32_t i = d >= 0 ? uint32_t(d) : uint32_t(int32_t(N) + d);
    if (i >= N || !((key[i / 32] >> (i % 32)) & 1u)) return 0u;
    return d >= 0 ? 0x3C00u : 0xBC00u;  // 1 or -1
}

// kScores: decryption (scores from b - a*s), else b += a*s.
template <bool kScores>
__global__ void __launch_bounds__(kKpThreads, 1) k_key_product(const __grid_constant__ KeyProductArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    KpShared &sh = *reinterpret_cast<KpShared *>(smem);
    uint8_t *table = smem + kHeader;
    uint8_t *stages = table + kp_table_bytes(a.N);
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t N = a.N, groups = N / 8, n_chunks = N / kChunkWords;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(&sh.a_full[s], kConvWarps);
            mbar_init(&sh.a_empty[s], 1);
        }
        for (uint32_t t = 0; t < 2; ++t) {
            mbar_init(&sh.acc_full[t], 1);
            mbar_init(&sh.acc_empty[t], 4);
        }
        mbar_init(&sh.drain, 1);
        sh.abort = 0;
        fence_mbar_init();
    }
    if (threadIdx.x < N / 32) sh.key[threadIdx.x] = a.key.w[threadIdx.x];
    if (warp == kMmaWarp) tmem_alloc(&sh.tmem_base, 2 * kTileMax);
    __syncthreads();
    // core matrix q, row n (a coefficient), element e (a mask word):
    // difference 8 (q - (groups - 1)) + n - e
    for (uint32_t x = threadIdx.x; x < (2 * groups - 1) * 8; x += kKpThreads) {
        const int32_t d = 8 * (int32_t(x / 8) - int32_t(groups - 1)) + int32_t(x % 8);
        uint32_t h[4];
#pragma unroll
        for (int32_t e = 0; e < 4; ++e)
            h[e] = kp_entry(sh.key, N, d - 2 * e) | (kp_entry(sh.key, N, d - 2 * e - 1) << 16);
        sts_v4(smem_addr(table + x * 16), h[0], h[1], h[2], h[3]);
    }
    // the two lanes of each quadrant without a digit stay zero
    for (uint32_t x = threadIdx.x; x < kStages * (kChunkWords / 8) * 8; x += kKpThreads) {
        const uint32_t m = 32 * ((x % 8) / 2) + 30 + x % 2;
        sts_v4(smem_addr(stages + (x / 8) * kGroupBytes + m * 16), 0, 0, 0, 0);
    }
    fence_proxy_async_smem();  // the table is read by the tensor cores (async proxy)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    const uint64_t my_items =
        a.items > blockIdx.x ? (a.items - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;  // items blockIdx.x + i * grid
    const uint32_t coef_pad = (a.n_coef + 15u) & ~15u;
    // columns of tile t of an item's pair: from n0, w of them (0: none)
    auto tile_of = [&](uint64_t item, uint32_t t, uint32_t &n0, uint32_t &w) {
        n0 = (2 * uint32_t(item % a.pairs) + t) * a.tile_cols;
        w = n0 < coef_pad ? min(a.tile_cols, coef_pad - n0) : 0u;
    };

    if (warp >= kConvWarp0) {
        // ---------------------------------------------------------- converters
        const uint32_t cid = threadIdx.x - 32 * kConvWarp0;
        const uint32_t l = cid % 8, row = cid / 8;  // group l of each chunk, rows `row` and `row + 20`
        const uint64_t total = my_items * n_chunks;
        uint64_t f_item = blockIdx.x;  // the next load's item and chunk
        uint32_t f_c = 0;
        const uint32_t *f_src[2];
        auto open = [&]() {
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint64_t r = (f_item / a.pairs) * kRows + row + h * (kRows / 2);
                f_src[h] = f_item < a.items && r < a.n_rows
                               ? reinterpret_cast<const uint32_t *>(kp_row(a, r)) + (N - 8 * (l + 1))
                               : nullptr;
            }
        };
        // the bodies of the item's rows, wanted by the epilogue after the item's
        // last chunk, on their way to L2
        auto prefetch_bodies = [&]() {
            const uint32_t lo = 2 * uint32_t(f_item % a.pairs) * a.tile_cols;
            const uint32_t hi = min(lo + 2 * a.tile_cols, a.n_coef);
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h)
                if (f_src[h])
                    for (uint32_t c = lo + 32 * l; c < hi; c += 256)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(f_src[h] + 8 * (l + 1) + c));
        };
        auto fetch = [&](uint32_t (&v)[2][8]) {
            if (f_c == 0) prefetch_bodies();
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                if (f_src[h]) {
                    kp_load<2>(f_src[h] - kChunkWords * f_c, a.vec_rows, v[h]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[h][e] = 0;
                }
            }
            if (++f_c == n_chunks) {
                f_c = 0;
                f_item += gridDim.x;
                open();
            }
        };
        open();
        uint32_t buf[2][2][8];
        fetch(buf[0]);
        fetch(buf[1]);
        bool ok = true;
        auto step = [&](uint64_t g, uint32_t (&v)[2][8]) {
            const uint32_t s = uint32_t(g % kStages);
            if (g >= kStages && !tc_warp_wait(&sh.abort, &sh.a_empty[s], uint32_t(g / kStages - 1) & 1u, a.err, lane))
                return false;
            const uint32_t dst = smem_addr(stages + s * kStageBytes) + l * kGroupBytes;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                uint32_t u[3][4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t x = v[h][2 * e], y = v[h][2 * e + 1];
                    u[0][e] = __byte_perm(x, y, 0x5410) & 0x07FF07FFu;
                    u[1][e] = __byte_perm(x >> 11, y >> 11, 0x5410) & 0x07FF07FFu;
                    u[2][e] = (__byte_perm(x, y, 0x7632) >> 6) & 0x03FF03FFu;
                }
                const uint32_t r = row + h * (kRows / 2), m = 32 * (r / 10) + r % 10;
#pragma unroll
                for (uint32_t d = 0; d < 3; ++d)
                    sts_v4(dst + (m + 10 * d) * 16, u[d][0], u[d][1], u[d][2], u[d][3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.a_full[s]);
            fetch(v);
            return true;
        };
        for (uint64_t g = 0; ok && g < total; g += 2) {
            ok = step(g, buf[0]);
            if (ok && g + 1 < total) ok = step(g + 1, buf[1]);
        }
    } else if (warp == kMmaWarp) {
        // ----------------------------------------------------------------- MMA
        const bool leader = elect_one();
        // where a tile is in the CTA's stream of chunks, and its columns
        struct Cursor {
            uint64_t i;  // item number
            uint32_t c, s, round;
            uint32_t w, idesc;
            uint64_t b;  // descriptor of the tile's next K-step
        } at[2] = {};
        const uint64_t a_desc = umma_desc(smem_addr(stages), kGroupBytes, 128);
        const uint32_t t_base = smem_addr(table);
        // tile t over its next chunk; false: a wait ended
        auto chunk = [&](uint32_t t, Cursor &x) {
            if (x.c == 0) {
                uint32_t n0;
                tile_of(blockIdx.x + x.i * gridDim.x, t, n0, x.w);
                x.idesc = umma_idesc_f16(128, x.w);
                x.b = umma_desc(t_base + n0 * 16, 128, 128);
                if (x.i > 0) {
                    if (!tc_wait(&sh.abort, &sh.acc_empty[t], uint32_t(x.i - 1) & 1u, a.err)) return false;
                    tc_fence_after();
                }
            }
            const uint64_t da = a_desc + x.s * (kStageBytes / 16);
            if (leader) {
                if (x.w) {
#pragma unroll
                    for (uint32_t j = 0; j < kChunkWords / 16; ++j)
                        umma_f16(tmem + t * kTileMax, da + j * (2 * kGroupBytes / 16), x.b + j * 16, x.idesc,
                                 x.c + j > 0 ? 1u : 0u);
                }
                if (t == 1) umma_commit(&sh.a_empty[x.s]);
                if (x.c + 1 == n_chunks) umma_commit(&sh.acc_full[t]);
            }
            __syncwarp();
            x.b += (kChunkWords / 8) * (128 / 16);
            if (++x.c == n_chunks) {
                x.c = 0;
                ++x.i;
            }
            if (++x.s == kStages) {
                x.s = 0;
                ++x.round;
            }
            return true;
        };
        bool ok = true;
        for (uint32_t lead = 0; ok && at[1].i < my_items; lead = min(lead + 1, kLag)) {
            if (at[0].i < my_items) {
                ok = tc_wait(&sh.abort, &sh.a_full[at[0].s], at[0].round & 1u, a.err);
                if (!ok) break;
                tc_fence_after();
                ok = chunk(0, at[0]);
            }
            if (ok && lead >= kLag) ok = chunk(1, at[1]);
        }
        // every MMA issued has completed before TMEM is released
        if (leader) umma_commit(&sh.drain);
        mbar_wait_bounded(&sh.drain, 0, nullptr);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        const uint32_t q = lane / 10, r = lane % 10;  // digit and row of this lane; q = 3: none
        const uint32_t mult = q < 3 ? 1u << (11 * q) : 0u;
        const uint32_t minus_magic = 0u - kMagicBits * mult;
        const uint32_t src_a = ((q + 1) % 3) * 10 + r, src_b = ((q + 2) % 3) * 10 + r;
        const uint32_t t = warp / 4, quadrant = warp % 4;
        for (uint64_t i = 0; i < my_items; ++i) {
            const uint64_t item = blockIdx.x + i * gridDim.x;
            const uint64_t row = (item / a.pairs) * kRows + 10 * quadrant + r;
            const bool has = q < 3 && row < a.n_rows;
            uint32_t n0, w;
            tile_of(item, t, n0, w);
            // this lane finishes columns 12 g + 4 q .. + 3 of the tile; the body
            // words of the next 48 columns are loaded while these are finished
            uint32_t *body = has ? reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(kp_row(a, row))) + N + n0 : nullptr;
            uint32_t *dst = kScores ? reinterpret_cast<uint32_t *>(a.scores) + row * a.n_coef + n0 : body;
            const uint32_t n_has = has ? min(w, a.n_coef - min(a.n_coef, n0)) : 0u;  // live columns
            uint32_t nb[4][4];
            auto load_body = [&](uint32_t c0) {
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
                    const uint32_t c = c0 + 12 * g + 4 * q;
                    if (c < n_has) kp_load<1>(body + c, a.vec_rows, nb[g]);
                }
            };
            load_body(0);
            if (!tc_warp_wait(&sh.abort, &sh.acc_full[t], uint32_t(i) & 1u, a.err, lane)) break;
            tc_fence_after();
            const uint32_t base = tmem + ((32 * quadrant) << 16) + t * kTileMax;
            for (uint32_t c0 = 0; c0 < w; c0 += 48) {
                uint32_t v[3][16];
                tmem_ld16(base + c0, v[0]);
                // blocks past the tile's end are not this tile's: read none of them
                if (c0 + 16 < w) tmem_ld16(base + c0 + 16, v[1]);
                if (c0 + 32 < w) tmem_ld16(base + c0 + 32, v[2]);
                tmem_wait_ld();
                uint32_t b[4][4];
#pragma unroll
                for (int e = 0; e < 16; ++e) b[e / 4][e % 4] = nb[e / 4][e % 4];
                load_body(c0 + 48);
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e) {
                        uint32_t x[3];
#pragma unroll
                        for (uint32_t k = 0; k < 3; ++k) {
                            const uint32_t at = 12 * g + 4 * k + e;
                            x[k] = __float_as_uint(__fadd_rn(__uint_as_float(v[at / 16][at % 16]), 0.75f)) * mult +
                                   minus_magic;
                        }
                        const uint32_t own = q == 0 ? x[0] : q == 1 ? x[1] : x[2];
                        const uint32_t to_a = q == 0 ? x[2] : q == 1 ? x[0] : x[1];
                        const uint32_t to_b = q == 0 ? x[1] : q == 1 ? x[2] : x[0];
                        const uint32_t p = own + __shfl_sync(0xFFFFFFFFu, to_a, src_a) +
                                           __shfl_sync(0xFFFFFFFFu, to_b, src_b);
                        if (kScores)
                            b[g][e] = __float_as_uint(__int2float_rn(int32_t(b[g][e] - p)) * 0x1p-32f);
                        else
                            b[g][e] += p;
                    }
                    const uint32_t c = c0 + 12 * g + 4 * q;
                    if (c + 4 <= n_has && (kScores ? a.vec_scores : a.vec_rows)) {
                        *reinterpret_cast<uint4 *>(dst + c) = make_uint4(b[g][0], b[g][1], b[g][2], b[g][3]);
                    } else {
#pragma unroll
                        for (uint32_t e = 0; e < 4; ++e)
                            if (c + e < n_has) dst[c + e] = b[g][e];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.acc_empty[t]);
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem, 2 * kTileMax);
}

}  // namespace

cudaError_t launch_key_product(KeyProductArgs a, int sm_count, cudaStream_t s) {
    if (a.n_rows == 0 || a.n_coef == 0) return cudaSuccess;
    if (!key_product_supported(a.N) || a.N % kChunkWords || a.n_coef > a.N) return cudaErrorInvalidValue;
    const uint64_t row_tiles = (a.n_rows + kRows - 1) / kRows;
    const uint32_t coef_pad = (a.n_coef + 15u) & ~15u;
    // Pairs of column tiles per 40 rows: as few as the accumulators allow (a
    // row's digits are split once per pair), more when there are fewer row
    // tiles than SMs, down to tiles of 32 columns.
    const uint32_t least = (coef_pad + 2 * kTileMax - 1) / (2 * kTileMax);
    const uint32_t most = std::max(least, (coef_pad + 63) / 64);
    const uint64_t want = uint64_t(sm_count) / row_tiles;
    uint32_t pairs = uint32_t(std::min<uint64_t>(most, std::max<uint64_t>(least, want)));
    a.tile_cols = ((coef_pad + 2 * pairs - 1) / (2 * pairs) + 15u) & ~15u;
    a.pairs = (coef_pad + 2 * a.tile_cols - 1) / (2 * a.tile_cols);
    a.items = row_tiles * a.pairs;
    a.vec_rows = ((reinterpret_cast<uintptr_t>(a.rows) | a.stride) & 15u) == 0;
    a.vec_scores = ((reinterpret_cast<uintptr_t>(a.scores) | (uint64_t(a.n_coef) * 4)) & 15u) == 0;
    auto *fn = a.scores ? k_key_product<true> : k_key_product<false>;
    fn<<<uint32_t(std::min<uint64_t>(a.items, uint64_t(sm_count))), kKpThreads, kp_smem(a.N), s>>>(a);
    return cudaGetLastError();
}

cudaError_t configure_key_product() {
    for (auto *fn : {k_key_product<true>, k_key_product<false>}) {
        const cudaError_t e =
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kp_smem(kKeyMaxN)));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace idash
