// Exact integer-polynomial x TRLWE scoring:
//   out_o = sum_f W_{o,f}(X) * C_f(X)  in Z/2^32[X]/(X^N + 1), on a and b,
// then b[s] += bias_o * one for s < num_samples and b[j] = 0 for
// j >= region_size, as the TRLWE form does (eval/idash.cpp:805-810, 839-841).
// The reference's own terms are the special case W = coef * X^(-r*REGION_SIZE)
// (eval/idash.cpp:817, 830-833); the only dense polynomial products in the
// reference are TFHE's double FFT inside encryption and decryption
// (eval/idash.cpp:625, 714), which cannot be exact here: a term is bounded by
// N * 2^13 * 2^31 = 2^54 and a 60-term sum by ~2^60, beyond 53 bits.
//
// Exactness: every coefficient's true integer value S (ciphertext words taken
// as signed 32-bit) satisfies |S| <= terms * max|W| * N * 2^31 < p1*p2 / 2,
// checked when the model is built.  S is computed modulo two NTT primes
// p1, p2 < 2^31 (p = 1 mod 2N) and recovered by CRT, then reduced mod 2^32.
//
// Kernels: k_ntt (model polynomials, once per model, and input TRLWE rows, once
// per call -> NTT, stored as centred residues) and k_intpoly_score (groups of
// outputs: pointwise multiply-accumulate over the terms as exact 64-bit sums,
// inverse NTT, CRT, epilogue).  Negacyclic NTTs are the Cooley-Tukey /
// Gentleman-Sande pair with bit-reversed powers of a primitive 2N-th root psi
// (Longa & Naehrig, CANS 2016).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "capi_internal.hpp"
#include "common.cuh"
#include "tcgen05.cuh"

namespace idash {

namespace {

constexpr uint32_t kPrimes[2] = {2147473409u, 2147389441u};  // both = 1 mod 2048
constexpr uint32_t kPsi2048[2] = {383167813u, 211808905u};   // primitive 2048-th roots of unity
constexpr int kNttThreads = 256;
constexpr uint32_t kIpN = 1024;  // polynomial size of the row and scoring kernels: 256 threads x 4 points

// 2^32 mod p is small for both primes (20478 and 188414), so folding the high
// word of a 64-bit sum onto the low one with it shrinks the sum below 2^49.
static_assert((uint64_t(1) << 32) % kPrimes[0] < (1u << 18) && (uint64_t(1) << 32) % kPrimes[1] < (1u << 18),
              "fold bound");

struct NttConsts {
    uint32_t p[2];
    uint32_t pinv[2];       // -p^-1 mod 2^32
    int32_t r1[2];          // R mod p, R = 2^32
    uint2 nscale[2];        // N^-1 * R mod p, the factor of the last inverse stage, for mul_lazy
    uint2 nscale_tw[2];     // nscale * (that stage's twiddle) mod p
    uint2 p1inv;            // p1^-1 mod p2
    uint64_t M, M_half;     // p1 * p2 and floor(M / 2)
};

uint64_t mulmod(uint64_t a, uint64_t b, uint64_t p) { return uint64_t((unsigned __int128)a * b % p); }
uint64_t powmod(uint64_t a, uint64_t e, uint64_t p) {
    uint64_t r = 1;
    for (a %= p; e; e >>= 1, a = mulmod(a, a, p))
        if (e & 1) r = mulmod(r, a, p);
    return r;
}

// x < 2p -> x mod p.
__device__ __forceinline__ uint32_t reduce_once(uint32_t x, uint32_t p) { return min(x, x - p); }

// v*S mod p, not fully reduced (below 2p), for any 32-bit v and S < p, with
// w = {S, floor(2^32 S / p)} (Shoup's product by a known factor; Harvey,
// "Faster arithmetic for number-theoretic transforms", 2014): one high and two
// low multiplications, 8 cycles of the multiplier a warp against 11 of a
// Montgomery product.
__device__ __forceinline__ uint32_t mul_lazy(uint32_t v, uint2 w, uint32_t p) { return v * w.x - __umulhi(v, w.y) * p; }

// Cooley-Tukey butterfly of the forward transform: (u, v) -> (u + v*S, u - v*S)
// for u < p and any v; results below p, or below 2p where kLazy: points that
// the next stage multiplies need no more.
template <bool kLazy>
__device__ __forceinline__ void ct_butterfly(uint32_t &u, uint32_t &v, uint2 S, uint32_t p) {
    const uint32_t w = reduce_once(mul_lazy(v, S, p), p);
    const uint32_t d = u - w;
    v = kLazy ? d + p : min(d, d + p);
    u = kLazy ? u + w : reduce_once(u + w, p);
}

// A residue x in [0, p) as the congruent value in (-p/2, p/2]: transforms are
// stored this way so that a product of two has magnitude below 2^60.
__device__ __forceinline__ int32_t centred(uint32_t x, uint32_t p) { return x > p / 2 ? int32_t(x - p) : int32_t(x); }

// Gentleman-Sande butterfly of the inverse transform: (u, v) -> (u + v, (u -
// v)*S), all below p.
__device__ __forceinline__ void gs_butterfly(uint32_t &u, uint32_t &v, uint2 S, uint32_t p) {
    const uint32_t d = u - v + p;
    u = reduce_once(u + v, p);
    v = reduce_once(mul_lazy(d, S, p), p);
}

// Stage i of five on 32 points in registers, and those after it: pairs points
// 16 >> i apart, its factor of group g at index 2^i + g of `tw` (two
// consecutive indices in 16 bytes, kStep 16-byte units from those to the next
// two).
template <uint32_t kStep, uint32_t i = 0>
__device__ __forceinline__ void ct_stages(uint32_t (&x)[32], const uint4 *tw, uint32_t p) {
    constexpr uint32_t h = 16u >> i;
    uint4 w{};
#pragma unroll
    for (uint32_t g = 0; g < (1u << i); ++g) {
        const uint32_t idx = (1u << i) + g;
        if (idx == 1 || idx % 2 == 0) w = tw[idx / 2 * kStep];
        const uint2 S = idx % 2 ? make_uint2(w.z, w.w) : make_uint2(w.x, w.y);
#pragma unroll
        for (uint32_t e = 2 * h * g; e < 2 * h * g + h; ++e) {
            if (e & (h / 2)) ct_butterfly<true>(x[e], x[e + h], S, p);
            else ct_butterfly<false>(x[e], x[e + h], S, p);
        }
    }
    if constexpr (i < 4) ct_stages<kStep, i + 1>(x, tw, p);
}

// The inverse's stages: stage a (to the last) pairs points 1 << a apart.
template <uint32_t kStep, uint32_t last, uint32_t a = 0>
__device__ __forceinline__ void gs_stages(uint32_t (&x)[32], const uint4 *tw, uint32_t p) {
    constexpr uint32_t t = 1u << a;
    uint4 w{};
#pragma unroll
    for (uint32_t g = 0; g < (16u >> a); ++g) {
        const uint32_t idx = (16u >> a) + g;
        if (idx == 1 || idx % 2 == 0) w = tw[idx / 2 * kStep];
        const uint2 S = idx % 2 ? make_uint2(w.z, w.w) : make_uint2(w.x, w.y);
#pragma unroll
        for (uint32_t e = 2 * t * g; e < 2 * t * g + t; ++e) gs_butterfly(x[e], x[e + t], S, p);
    }
    if constexpr (a < last) gs_stages<kStep, last, a + 1>(x, tw, p);
}

// Factors of a 1024-point transform as two passes of 32 points, in shared
// memory, from tw[prime][N].  The pass over points 32 or more apart uses
// factors 1 .. 31 for every lane; in the other, lane L has points 32L .. 32L +
// 31 and uses factor ((32 + L) << i) + g for group g of the stage with 2^i
// groups.
struct TwTables {
    uint4 far[2][16];        // [prime][index / 2]
    uint4 near[2][16][32];   // [prime][index / 2][lane]
};
__device__ __forceinline__ void load_tables(TwTables &t, const uint2 *tw) {
    uint2 *far = reinterpret_cast<uint2 *>(t.far), *near = reinterpret_cast<uint2 *>(t.near);
    for (uint32_t x = threadIdx.x; x < 64; x += blockDim.x) far[x] = tw[(x / 32) * kIpN + x % 32];
    for (uint32_t x = threadIdx.x; x < 2 * kIpN; x += blockDim.x) {
        const uint32_t q = x / kIpN, idx = x % kIpN / 64 * 2 + x % 2, lane = x / 2 % 32;
        const uint32_t i = idx ? 31u - uint32_t(__clz(int(idx))) : 0u;  // index 2^i + g; 0 is not used
        near[x] = idx ? tw[q * kIpN + ((32 + lane) << i) + idx - (1u << i)] : make_uint2(0, 0);
    }
}

// A warp's 1024 words in shared memory: 32 rows of 32, 16-byte piece p of row
// r at piece p ^ (r % 8), so that both a column (point 32e + lane) and a row
// (points 32 lane + e) go without bank conflicts.
__device__ __forceinline__ void put_columns(uint32_t addr, uint32_t lane, const uint32_t (&x)[32]) {
    const uint32_t a = addr + lane * 4;
#pragma unroll
    for (uint32_t e = 0; e < 32; ++e)
        asm volatile("st.shared.u32 [%0], %1;" ::"r"((a ^ ((e % 8) * 16)) + e * 128), "r"(x[e]) : "memory");
}
__device__ __forceinline__ void get_rows(uint32_t addr, uint32_t lane, uint32_t (&x)[32]) {
    const uint32_t a = addr + lane * 128 + (lane % 8) * 16;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint4 v = lds_v4(a ^ (k * 16));
        x[4 * k] = v.x;
        x[4 * k + 1] = v.y;
        x[4 * k + 2] = v.z;
        x[4 * k + 3] = v.w;
    }
}
__device__ __forceinline__ void put_rows(uint32_t addr, uint32_t lane, const uint32_t (&x)[32]) {
    const uint32_t a = addr + lane * 128 + (lane % 8) * 16;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a ^ (k * 16)), "r"(x[4 * k]), "r"(x[4 * k + 1]),
                     "r"(x[4 * k + 2]), "r"(x[4 * k + 3])
                     : "memory");
}

__device__ __forceinline__ void get_columns(uint32_t addr, uint32_t lane, uint32_t (&x)[32]) {
    const uint32_t a = addr + lane * 4;
#pragma unroll
    for (uint32_t e = 0; e < 32; ++e)
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x[e]) : "r"((a ^ ((e % 8) * 16)) + e * 128) : "memory");
}

// Where a weight polynomial's transforms go, in units of N words: the first
// prime's, and (plus one) how far from it the second's is (k_intpoly_score
// reads the weights of a group's outputs at one term in one piece).
constexpr uint32_t kSlotBits = 30;
constexpr uint32_t ip_slot(uint64_t at, uint32_t members) { return uint32_t(at) | ((members - 1) << kSlotBits); }

// Forward transforms of 1024-point polynomials, stored as centred residues.
// Polynomial i of model weights (int16): at in + i * N * 2, stored at slots[i];
// coefficients beyond max_abs break the exactness bound and are reported.  Of
// input rows (signed words): half i % 2 of row i / 2, rows `stride` bytes
// apart, stored [row][prime][half][N].
//
// One warp per polynomial and prime.  A lane holds 32 points: five stages on
// points lane + 32e in registers, one exchange through the warp's own shared
// memory, five stages on points 32 lane + e, and an exchange back so that
// global stores are whole rows; no barrier across warps.  The integer pipes
// bound it (72% busy with the multiplier, 59% with additions and minima).
// 90,540 weight polynomials: 0.372 ms (0.93 GB, 2.5 TB/s), 1.668 ms with a
// block per polynomial and a pass through shared memory per stage, 0.420 ms
// with Montgomery products.
template <typename Word>
__global__ void __launch_bounds__(kNttThreads, sizeof(Word) == 2 ? 3 : 2)
    k_ntt(const uint8_t *in, uint64_t stride, uint64_t n_polys, const uint2 *tw, NttConsts k, int32_t max_abs,
          const uint32_t *slots, uint32_t *hat, uint32_t *err) {
    constexpr bool kModel = sizeof(Word) == 2;
    __shared__ TwTables tables;
    __shared__ __align__(1024) uint32_t exchange[kNttThreads / 32][kIpN];
    load_tables(tables, tw);
    __syncthreads();
    const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const uint32_t mine = smem_addr(exchange[warp]);
    // few polynomials spread over the SMs before they fill one
    const uint64_t step = uint64_t(gridDim.x) * (kNttThreads / 32);
    for (uint64_t j = blockIdx.x + uint64_t(gridDim.x) * warp; j < 2 * n_polys; j += step) {
        const uint64_t i = j / 2;
        const uint32_t q = uint32_t(j % 2), p = q ? k.p[1] : k.p[0];
        const Word *src = reinterpret_cast<const Word *>(kModel ? in + i * (kIpN * 2)
                                                                : in + (i / 2) * stride + (i % 2) * (kIpN * 4)) + lane;
        const uint32_t slot = kModel ? slots[i] : 0;
        const uint64_t at = kModel ? slot & ((1u << kSlotBits) - 1) : (i / 2) * 4 + i % 2;
        const uint32_t apart = kModel ? (slot >> kSlotBits) + 1 : 2;
        uint4 *dst = reinterpret_cast<uint4 *>(hat + (at + q * apart) * kIpN) + lane;
        uint32_t x[32];
        bool bad = false;
#pragma unroll
        for (uint32_t e = 0; e < 32; ++e) {
            const int32_t v = src[32 * e];
            if (kModel) {
                bad |= v > max_abs || v < -max_abs;
                x[e] = uint32_t(v < 0 ? v + int32_t(p) : v);
            } else {
                x[e] = uint32_t(v) + (v < 0 ? 2 * p : 0u);  // below 2p
                if (e < 16) x[e] = reduce_once(x[e], p);
            }
        }
        if (kModel && bad) report_error(err, kDevBadIndex);
        ct_stages<1>(x, tables.far[q], p);
        __syncwarp();  // the rows read last are out of the buffer
        put_columns(mine, lane, x);
        __syncwarp();
        get_rows(mine, lane, x);
        ct_stages<32>(x, &tables.near[q][0][lane], p);
#pragma unroll
        for (uint32_t e = 0; e < 32; ++e) x[e] = uint32_t(centred(x[e], p));
        __syncwarp();
        put_rows(mine, lane, x);
        __syncwarp();
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {  // 16-byte piece 32r + lane: row 4r + lane / 8
            const uint32_t row = 4 * r + lane / 8;
            dst[32 * r] = lds_v4(mine + row * 128 + ((lane % 8) ^ (row % 8)) * 16);
        }
    }
}

struct IntpolyArgs {
    const uint64_t *term_ptr;
    const uint32_t *term_row;
    const uint64_t *group_first;  // group g: outputs [group_first[g], group_first[g + 1])
    uint64_t group_begin, group_end;  // groups scored by this launch
    const uint32_t *w_hat;
    const uint32_t *c_hat;
    const int32_t *bias;
    const uint2 *itw;
    NttConsts k;
    uint32_t N, num_samples, region_size, n_rows;
    int32_t one;
    uint64_t out_begin, out_end;  // outputs written (output o -> row o - out_begin)
    uint8_t *out;  // payload of output row 0
    uint64_t out_stride;
    uint32_t *err;
};

constexpr uint32_t kGroupMax = 3;     // outputs sharing one term-row list (a target's genotypes)
// k_intpoly_score: a consumer thread has four points of one prime
constexpr uint32_t kConsumers = kIpN / 2;
constexpr uint32_t kIpEpiWarps = 2 * kGroupMax;                       // one per output and polynomial
constexpr uint32_t kScoreBlock = kConsumers + 32 * kIpEpiWarps + 64;  // and a producer warp per prime
constexpr uint32_t kScoreStages = 8;                                  // half row steps (one prime) in flight per CTA
// Products of centred residues have magnitude below 2^60; a folded sum is
// below 2^49, so kFoldSteps products more stay below 2^63.
constexpr uint32_t kFoldSteps = 7;

// hi * 2^32 + lo  ->  hi * (2^32 mod p) + lo: same residue, magnitude < 2^49
// for |T| < 2^63.  In place on the halves: written as an expression, it made
// the compiler copy the sums at every step (a row step of 24 sums a thread
// went from 526 to 1,010 cycles).
__device__ __forceinline__ void fold(int64_t &T, int32_t r1) {
    uint32_t lo = uint32_t(T), hi = uint32_t(uint64_t(T) >> 32);
    asm("{\n\t.reg .b32 h;\n\tmov.b32 h, %1;\n\t"
        "mad.lo.cc.u32 %0, h, %2, %0;\n\tmadc.hi.s32 %1, h, %2, 0;\n\t}"
        : "+r"(lo), "+r"(hi)
        : "r"(r1));
    T = int64_t((uint64_t(hi) << 32) | lo);
}

// The epilogue's wait for a group's sums is as long as the group: up to 2^20 row
// steps, 0.44 s of the second that other waits have.  So its limit grows by this
// for each step (a step takes some 1,100 cycles with all SMs at work).
constexpr long long kStepLimitCycles = 1 << 14;

// Stage layout, for one prime: the input row's transform (2 polynomials), then
// the weights' of up to kGroupMax outputs at the same term, N words each.
constexpr uint32_t kStageWords = (2 + kGroupMax) * kIpN;
struct IpHeader {
    uint64_t full[kScoreStages], empty[kScoreStages];
    uint64_t sums_full, sums_empty;  // a group's sums
    uint32_t info[kScoreStages];     // of a group's first stage: kIp* bits, 4 * its row steps
    uint32_t abort;
};
constexpr uint32_t kIpEmpty = 1, kIpFinal = 2;  // one step without a row; the CTA's last group
constexpr uint32_t kIpHeader = 256;
static_assert(sizeof(IpHeader) <= kIpHeader, "header area");
constexpr uint32_t kSumWords = 4 * kGroupMax * kIpN;  // [output][poly][prime][N]
constexpr size_t kIpScoreSmem =
    kIpHeader + 4 * (size_t(kScoreStages) * kStageWords + kSumWords) + sizeof(TwTables);
static_assert(kIpScoreSmem <= 227 * 1024, "shared memory of k_intpoly_score");

// One row step of a consumer thread: adds the products of four points, for
// both polynomials of kGroupMax outputs (the sums of outputs that a group does
// not have are not used; a branch per group size made the compiler copy the 48
// registers of sums at every step).  `at`: the thread's words of the stage.
__device__ __forceinline__ void ip_accumulate(int64_t (&acc)[kGroupMax][2][4], uint32_t at) {
    const uint4 c[2] = {lds_v4(at), lds_v4(at + kIpN * 4)};
#pragma unroll
    for (uint32_t m = 0; m < kGroupMax; ++m) {
        const uint4 w = lds_v4(at + (2 + m) * kIpN * 4);
#pragma unroll
        for (uint32_t poly = 0; poly < 2; ++poly) {
            // one widening multiply-add each; as mad.wide in inline assembly a
            // product and two additions
            int64_t *t = acc[m][poly];
            t[0] += int64_t(int32_t(w.x)) * int32_t(c[poly].x);
            t[1] += int64_t(int32_t(w.y)) * int32_t(c[poly].y);
            t[2] += int64_t(int32_t(w.z)) * int32_t(c[poly].z);
            t[3] += int64_t(int32_t(w.w)) * int32_t(c[poly].w);
        }
    }
}

// Persistent, one CTA per SM over output groups: the outputs of a group read
// the same input rows in the same order (normally the three genotype outputs
// of a target), so each row step brings one input transform (16 KiB) and one
// weight transform (8 KiB) per output, half of either for each prime.  Roles:
//   producers   (one warp a prime) keep kScoreStages half steps in flight
//               with cp.async.bulk into a ring, across group boundaries;
//   consumers   (8 warps a prime) a thread takes four points of every output
//               of the group, so that the input transform is read from shared
//               memory once for all of them.  A product is one signed widening
//               multiplication and a 64-bit sum; every kFoldSteps terms the
//               sums are folded with 2^32 mod p, which keeps them exact
//               without a reduction per product.  The residues (times 2^-32)
//               go to shared memory, and the next group begins;
//   epilogue    (6 warps) one per output and polynomial: the inverse
//               transforms of both primes as two passes of 32 points in
//               registers, CRT, bias and zeroed coefficients, while the
//               consumers are at the next group.
// Memory bounds it: 540,000 terms (4.4 GB of weights, 3 GB of input transforms
// from L2) take 0.70 ms, 0.65 ms with the sums and the epilogue left out, and
// took 0.93 ms with the inverse transforms between the groups, one thread for
// both primes' copies and each output's sums reading the input transform anew.
// Waiting consumers poll each for itself: meeting at a named barrier cost 8%.
// Every wait is bounded and ends early once another role gave up; the producers
// let their copies in flight land before they return, however they came there.
__global__ void __launch_bounds__(kScoreBlock, 1) k_intpoly_score(const IntpolyArgs a) {
    extern __shared__ __align__(1024) uint8_t ip_smem[];
    constexpr uint32_t N = kIpN;  // a.N, checked on the host
    IpHeader &sh = *reinterpret_cast<IpHeader *>(ip_smem);
    TwTables &tables = *reinterpret_cast<TwTables *>(ip_smem + kIpHeader);
    uint32_t *stage_words = reinterpret_cast<uint32_t *>(ip_smem + kIpHeader + sizeof(TwTables));
    const uint32_t stage0 = smem_addr(stage_words);
    const uint32_t sums = stage0 + kScoreStages * kStageWords * 4;  // whole rows of 128 bytes
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    if (tid == 0) {
        for (uint32_t s = 0; s < kScoreStages; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], kConsumers / 64);
        }
        mbar_init(&sh.sums_full, kConsumers / 32);
        mbar_init(&sh.sums_empty, kIpEpiWarps);
        sh.abort = 0;
        fence_mbar_init();
    }
    load_tables(tables, a.itw);
    __syncthreads();

    if (warp < kConsumers / 32) {
        // ----------------------------------------------------------- consumers
        const uint32_t q = warp / (kConsumers / 64), pt = tid % (kConsumers / 2);  // prime, points 4 pt ..
        const uint32_t p = q ? a.k.p[1] : a.k.p[0], pinv = q ? a.k.pinv[1] : a.k.pinv[0];
        const int32_t r1 = q ? a.k.r1[1] : a.k.r1[0];
        // A lane that gives up exits; the warp's barriers are for the others.
        uint32_t s = q, parity = 0;  // the prime's stages in turn: q, q + 2, ...
        const uint32_t base = stage0 + 16 * pt;
        for (uint32_t turn = 0;;) {
            int64_t acc[kGroupMax][2][4];  // [output][poly][point]
#pragma unroll
            for (uint32_t e = 0; e < kGroupMax * 8; ++e) acc[e / 8][e / 4 % 2][e % 4] = 0;
            if (!tc_wait(&sh.abort, &sh.full[s], parity, a.err)) return;
            const uint32_t info = reinterpret_cast<volatile uint32_t *>(sh.info)[s];
            uint32_t left = info / 4;  // row steps of the group
            const bool empty = info & kIpEmpty;
            while (left > 0) {
                // the step's data is here; kFoldSteps at most before a fold
                const uint32_t stop = left > kFoldSteps ? left - kFoldSteps : 0;
                for (;;) {
                    if (!empty) ip_accumulate(acc, base + s * (kStageWords * 4));
                    __syncwarp();  // this warp is done with the stage
                    if (lane == 0) mbar_arrive(&sh.empty[s]);
                    s += 2;
                    if (s >= kScoreStages) {
                        s -= kScoreStages;
                        parity ^= 1u;
                    }
                    if (--left > 0 && !tc_wait(&sh.abort, &sh.full[s], parity, a.err)) return;
                    if (left == stop) break;
                }
#pragma unroll
                for (uint32_t e = 0; e < kGroupMax * 8; ++e)
                    fold(acc[e / 8][e / 4 % 2][e % 4], r1);
            }

            if (turn > 0 && !tc_wait(&sh.abort, &sh.sums_empty, (turn - 1) & 1u, a.err)) return;
            ++turn;
            const uint32_t row = pt / 8;
            const uint32_t to = sums + q * (N * 4) + row * 128 + ((pt % 8) ^ (row % 8)) * 16;
#pragma unroll
            for (uint32_t m = 0; m < kGroupMax; ++m)
#pragma unroll
                for (uint32_t poly = 0; poly < 2; ++poly) {
                    uint32_t v[4];
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e) {
                        // a folded sum, lifted by p * 2^19 to a positive T < p * 2^32; T * 2^-32 mod p
                        const uint64_t T = uint64_t(acc[m][poly][e] + (int64_t(p) << 19));
                        const uint32_t f = uint32_t(T) * pinv;
                        v[e] = reduce_once(uint32_t((T + uint64_t(f) * p) >> 32), p);
                    }
                    sts_v4(to + (4 * m + 2 * poly) * N * 4, v[0], v[1], v[2], v[3]);
                }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.sums_full);
            if (info & kIpFinal) break;
        }
    } else if (warp < kConsumers / 32 + kIpEpiWarps) {
        // ------------------------------------------------------------ epilogue
        // Inverse transform (Gentleman-Sande; the stage of span t pairs points
        // j and j + t with twiddle itw[N / (2t) + j / (2t)]).
        const uint32_t m = (warp - kConsumers / 32) / 2, poly = (warp - kConsumers / 32) % 2;
        const uint32_t p0 = a.k.p[0], p1 = a.k.p[1];
        uint32_t turn = 0;
        uint64_t g = a.group_begin + blockIdx.x;
        for (; g < a.group_end; g += gridDim.x, ++turn) {
            const uint64_t o0 = a.group_first[g], o = o0 + m;
            const bool mine = o < a.group_first[g + 1] && o >= a.out_begin && o < a.out_end;
            const uint32_t add = mine && poly == 1 && a.bias ? uint32_t(a.bias[o]) * uint32_t(a.one) : 0u;
            const bool polls = m == 0 && poly == 0 && lane == 0;
            const long long limit =
                kWaitLimitCycles + (polls ? (long long)(a.term_ptr[o0 + 1] - a.term_ptr[o0]) * kStepLimitCycles : 0);
            if (!tc_team_wait<32 * kIpEpiWarps>(1, polls, &sh.abort, &sh.sums_full, turn & 1u, a.err, limit)) return;
            if (!mine) {
                if (lane == 0) mbar_arrive(&sh.sums_empty);
                continue;
            }
            uint32_t x[32];
            const uint32_t first = sums + (4 * m + 2 * poly) * N * 4;
#pragma unroll 1
            for (uint32_t q = 0; q < 2; ++q) {
                const uint32_t p = q ? p1 : p0;
                const uint32_t at = first + q * N * 4;
                get_rows(at, lane, x);
                gs_stages<32, 4>(x, &tables.near[q][0][lane], p);
                put_rows(at, lane, x);
                __syncwarp();
                get_columns(at, lane, x);
                gs_stages<1, 3>(x, tables.far[q], p);
                // the last stage, scaled by N^-1 * 2^32 (which also undoes the sums' factor)
                const uint2 s0 = q ? a.k.nscale[1] : a.k.nscale[0], s1 = q ? a.k.nscale_tw[1] : a.k.nscale_tw[0];
#pragma unroll
                for (uint32_t e = 0; e < 16; ++e) {
                    const uint32_t d = x[e] - x[e + 16] + p;
                    x[e] = reduce_once(mul_lazy(x[e] + x[e + 16], s0, p), p);
                    x[e + 16] = reduce_once(mul_lazy(d, s1, p), p);
                }
                if (q == 0) put_columns(at, lane, x);  // what this lane read, back to where it was
            }
            uint32_t *dst = reinterpret_cast<uint32_t *>(a.out + (o - a.out_begin) * a.out_stride) + poly * N + lane;
#pragma unroll
            for (uint32_t e = 0; e < 32; ++e) {
                // CRT: v = y + p1 * ((x - y) / p1 mod p2), signed, then mod 2^32
                uint32_t y;
                asm volatile("ld.shared.u32 %0, [%1];"
                             : "=r"(y)
                             : "r"(((first + lane * 4) ^ ((e % 8) * 16)) + e * 128)
                             : "memory");
                const uint32_t d = x[e] - reduce_once(y, p1) + p1;
                const uint32_t t = reduce_once(mul_lazy(d, a.k.p1inv, p1), p1);
                const uint64_t v = uint64_t(y) + uint64_t(p0) * t;
                uint32_t w = uint32_t(v);
                if (v > a.k.M_half) w -= uint32_t(a.k.M);
                if (poly == 1) {
                    const uint32_t j = 32 * e + lane;
                    if (j < a.num_samples) w += add;
                    if (j >= a.region_size) w = 0;
                }
                dst[32 * e] = w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.sums_empty);
        }
    } else {
        // ----------------------------------------------------------- producers
        // Lookups run ahead of the copies: a group's outputs two groups, its
        // terms one, a row one step.  The warp runs the loop whole and one
        // thread issues, so that addresses stay in uniform registers; each lane
        // leaves by its own verdict, as nothing in the loop waits for the others.
        const uint32_t q = warp - (kConsumers / 32 + kIpEpiWarps);
        const bool leader = elect_one();
        uint64_t g = a.group_begin + blockIdx.x;
        const uint64_t last = a.group_end - 1;
        uint64_t o0 = a.group_first[g], o1 = a.group_first[g + 1];
        uint64_t t0 = a.term_ptr[o0], t1 = a.term_ptr[o0 + 1];
        uint32_t members = uint32_t(o1 - o0), row = t1 > t0 ? a.term_row[t0] : 0;
        uint64_t ahead = min(g + gridDim.x, last);
        o0 = a.group_first[ahead];
        o1 = a.group_first[ahead + 1];
        uint32_t s = q, parity = 1, issued = 0;  // the prime's stages in turn: q, q + 2, ...
        bool ok = true;
        for (; ok && g < a.group_end; g += gridDim.x) {
            const uint64_t next_t0 = a.term_ptr[o0], next_t1 = a.term_ptr[o0 + 1];
            const uint32_t next_members = uint32_t(o1 - o0);
            ahead = min(ahead + gridDim.x, last);
            o0 = a.group_first[ahead];
            o1 = a.group_first[ahead + 1];
            const uint32_t n = uint32_t(t1 - t0), steps = n ? n : 1;  // an empty group: one step without copies
            const uint32_t info = 4 * steps | (n ? 0u : kIpEmpty) | (g + gridDim.x >= a.group_end ? kIpFinal : 0u);
            const uint32_t w_bytes = members * N * 4;
            const uint8_t *w = reinterpret_cast<const uint8_t *>(a.w_hat + t0 * (2 * N)) + q * w_bytes;
            const uint32_t *rows = a.term_row + t0;
            uint32_t next_row = 0;
            for (uint32_t i = 1; i <= steps; ++i) {
                uint32_t r = row;
                if (i < n) row = rows[i];
                else if (next_t1 > next_t0) next_row = a.term_row[next_t0];
                if (r >= a.n_rows) {
                    report_error(a.err, kDevBadIndex);
                    r = 0;  // read a valid row; the output is reported invalid
                }
                // a stage's first fill passes at once: the phase before the first counts as complete
                if (!(ok = tc_wait(&sh.abort, &sh.empty[s], parity, a.err))) break;
                if (leader) {
                    reinterpret_cast<volatile uint32_t *>(sh.info)[s] = info;
                    if (n) {
                        uint32_t *st = stage_words + s * kStageWords;
                        fence_proxy_async_smem();
                        mbar_arrive_expect_tx(&sh.full[s], 2 * N * 4 + w_bytes);
                        bulk_g2s(st, a.c_hat + uint64_t(r) * (4 * N) + q * (2 * N), 2 * N * 4, &sh.full[s]);
                        bulk_g2s(st + 2 * N, w, w_bytes, &sh.full[s]);
                    } else {
                        mbar_arrive(&sh.full[s]);
                    }
                }
                w += 2 * w_bytes;
                ++issued;
                s += 2;
                if (s >= kScoreStages) {
                    s -= kScoreStages;
                    parity ^= 1u;
                }
            }
            t0 = next_t0;
            t1 = next_t1;
            members = next_members;
            row = next_row;
        }
        if (leader) {
            // let the last copies land, also when the consumers give up once all are issued
            constexpr uint32_t kMine = kScoreStages / 2;
            for (uint32_t k = issued > kMine ? issued - kMine : 0; k < issued; ++k)
                mbar_wait_bounded(&sh.full[q + 2 * (k % kMine)], (k / kMine) & 1u, nullptr);
        }
    }
}

__global__ void k_synth_int16(uint64_t seed, uint64_t n, int32_t max_abs, int16_t *out) {
    const uint64_t key = mix64(seed + mix64(15));
    const uint32_t span = uint32_t(2 * max_abs);
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        out[i] = int16_t(int32_t(uint32_t(mix64(key ^ i) >> 32) % span) - max_abs);
}

// A factor and its quotient, for mul_lazy.
uint2 factor(uint64_t f, uint64_t p) { return make_uint2(uint32_t(f), uint32_t((f << 32) / p)); }

NttConsts make_consts(uint32_t N) {
    NttConsts k{};
    for (int q = 0; q < 2; ++q) {
        const uint64_t p = kPrimes[q];
        k.p[q] = uint32_t(p);
        uint32_t inv = 1;  // Newton iteration for p^-1 mod 2^32
        for (int it = 0; it < 5; ++it) inv *= 2u - uint32_t(p) * inv;
        k.pinv[q] = 0u - inv;
        const uint64_t R = (uint64_t(1) << 32) % p;
        k.r1[q] = int32_t(R);
        const uint64_t nscale = mulmod(powmod(N, p - 2, p), R, p);
        k.nscale[q] = factor(nscale, p);
        // the last inverse stage's twiddle: psi^-(N/2) (bit-reversed index 1)
        const uint64_t psi = powmod(kPsi2048[q], 2048 / (2 * N), p);
        k.nscale_tw[q] = factor(mulmod(powmod(powmod(psi, p - 2, p), N / 2, p), nscale, p), p);
    }
    const uint64_t p0 = kPrimes[0], p1 = kPrimes[1];
    k.p1inv = factor(powmod(p0 % p1, p1 - 2, p1), p1);
    k.M = p0 * p1;
    k.M_half = k.M / 2;
    return k;
}

// Bit-reversed powers of psi (forward) and psi^-1 (inverse), [prime][N] each,
// with their quotients.  psi is a primitive 2N-th root: psi_2048^(2048 / 2N).
void make_twiddles(uint32_t N, std::vector<uint2> *fwd, std::vector<uint2> *inv) {
    uint32_t logn = 0;
    while ((1u << logn) < N) ++logn;
    fwd->assign(2 * N, make_uint2(0, 0));
    inv->assign(2 * N, make_uint2(0, 0));
    for (int q = 0; q < 2; ++q) {
        const uint64_t p = kPrimes[q];
        const uint64_t psi = powmod(kPsi2048[q], 2048 / (2 * N), p);
        const uint64_t psi_inv = powmod(psi, p - 2, p);
        for (uint32_t i = 0; i < N; ++i) {
            uint32_t rev = 0;
            for (uint32_t b = 0; b < logn; ++b)
                if (i & (1u << b)) rev |= 1u << (logn - 1 - b);
            (*fwd)[q * N + i] = factor(powmod(psi, rev, p), p);
            (*inv)[q * N + i] = factor(powmod(psi_inv, rev, p), p);
        }
    }
}

}  // namespace

struct IntpolyModel {
    uint32_t N = 0, num_samples = 0, region_size = 0;
    int32_t one = 0, max_abs = 0;
    uint64_t n_out = 0, n_terms = 0, n_rows = 0;
    NttConsts k{};
    uint64_t *d_term_ptr = nullptr;
    uint32_t *d_term_row = nullptr;
    uint32_t *d_slot = nullptr;  // where each term's transform goes (ip_slot)
    // Output groups: consecutive outputs (at most kGroupMax) with identical
    // term-row lists; group g is outputs [group_first[g], group_first[g + 1]).
    std::vector<uint64_t> group_first;
    uint64_t *d_group_first = nullptr;
    int32_t *d_bias = nullptr;
    uint32_t *d_w_hat = nullptr;
    uint2 *d_tw = nullptr;   // forward twiddles and quotients [2][N]
    uint2 *d_itw = nullptr;  // inverse twiddles and quotients [2][N]
    uint32_t *d_c_hat = nullptr;
    uint64_t c_hat_rows = 0;
    std::mutex order;              // calls take their turns (IntpolyTurn)
    cudaEvent_t used = nullptr;    // the last call's kernels are done
    ~IntpolyModel() {
        if (used) cudaEventDestroy(used);
        cudaFree(d_term_ptr);
        cudaFree(d_term_row);
        cudaFree(d_slot);
        cudaFree(d_group_first);
        cudaFree(d_bias);
        cudaFree(d_w_hat);
        cudaFree(d_tw);
        cudaFree(d_itw);
        cudaFree(d_c_hat);
    }
};

namespace {

uint32_t ntt_grid(uint64_t n_polys, uint32_t per_sm, const idash_ctx *ctx) {
    return uint32_t(std::min<uint64_t>(n_polys, uint64_t(ctx->sm_count) * per_sm));
}

// A call's turn at the model's transforms, of which there is one set (d_w_hat,
// d_c_hat): its kernels follow those of the call before, whatever the streams.
// Captured into a caller's graph, the wait and the record are nodes of it, and a
// replay takes its turn like a call.
class IntpolyTurn {
    IntpolyModel &ip;
    cudaStream_t stream;
    std::lock_guard<std::mutex> lock;
    bool captured = false;

  public:
    IntpolyTurn(IntpolyModel &ip_, cudaStream_t s) : ip(ip_), stream(s), lock(ip_.order) {}
    cudaError_t begin() {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        const cudaError_t e = cudaStreamIsCapturing(stream, &status);
        if (e != cudaSuccess) return e;
        captured = status == cudaStreamCaptureStatusActive;
        return cudaStreamWaitEvent(stream, ip.used, captured ? cudaEventWaitExternal : cudaEventWaitDefault);
    }
    cudaError_t end() {
        return cudaEventRecordWithFlags(ip.used, stream, captured ? cudaEventRecordExternal : cudaEventRecordDefault);
    }
};

// The transforms of terms [t0, t0 + n), whose polynomials are at w.
cudaError_t launch_ntt_model(const IntpolyModel &ip, const int16_t *w, uint64_t t0, uint64_t n, idash_ctx *ctx,
                             cudaStream_t stream) {
    k_ntt<int16_t><<<ntt_grid(2 * n, 3, ctx), kNttThreads, 0, stream>>>(
        reinterpret_cast<const uint8_t *>(w), 0, n, ip.d_tw, ip.k, ip.max_abs, ip.d_slot + t0, ip.d_w_hat, ctx->d_err);
    return cudaGetLastError();
}

}  // namespace

}  // namespace idash

using namespace idash;

void idash_model::free_intpoly() {
    delete intpoly;
    intpoly = nullptr;
}

extern "C" idash_status idash_model_intpoly(idash_ctx *ctx, idash_model **model, const idash_intpoly_params *p,
                                            uint64_t n_out, const uint64_t *term_ptr, const uint32_t *term_feat,
                                            const int32_t *bias, uint64_t n_in_rows, const int16_t *term_poly,
                                            int term_poly_on_device) {
    if (!ctx || !model || !p || (n_out && !term_ptr)) return IDASH_ERR_INVALID_ARGUMENT;
    *model = nullptr;
    if (p->N != kIpN)
        return ctx->fail(IDASH_ERR_UNSUPPORTED, "the integer-polynomial kernels are built for N = 1024");
    if (p->num_samples > p->region_size || p->region_size > p->N)
        return ctx->fail(IDASH_ERR_INVALID_ARGUMENT, "need num_samples <= region_size <= N");
    if (p->max_abs_coef <= 0 || p->max_abs_coef > 32767)
        return ctx->fail(IDASH_ERR_INVALID_ARGUMENT, "max_abs_coef must be in [1, 32767]");
    const uint64_t nnz = n_out ? term_ptr[n_out] : 0;
    if (nnz >> (kSlotBits - 1)) return ctx->fail(IDASH_ERR_OUT_OF_MEMORY, "the weights' transforms exceed 4 TiB");
    if (nnz && (!term_feat || !term_poly)) return IDASH_ERR_INVALID_ARGUMENT;
    const NttConsts k = make_consts(p->N);
    // exactness: terms * max|W| * N * 2^31 < M / 2 for every output
    const double cap = double(k.M_half) / (double(p->max_abs_coef) * p->N * 2147483648.0);
    for (uint64_t o = 0; o < n_out; ++o) {
        if (term_ptr[o + 1] < term_ptr[o]) return ctx->fail(IDASH_ERR_INVALID_ARGUMENT, "term_ptr not monotone");
        if (double(term_ptr[o + 1] - term_ptr[o]) >= cap)
            return ctx->fail(IDASH_ERR_UNSUPPORTED, "output " + std::to_string(o) + " has too many terms for an "
                                                    "exact two-prime product at this max_abs_coef");
    }
    for (uint64_t t = 0; t < nnz; ++t)
        if (term_feat[t] >= n_in_rows) return ctx->fail(IDASH_ERR_INDEX, "a term names a row outside the input");

    idash_model *m = new idash_model();
    m->ctx = ctx;
    m->form = Form::kIntPoly;
    m->n_out = n_out;
    m->n_in_rows = n_in_rows;
    m->intpoly = new IntpolyModel();
    IntpolyModel &ip = *m->intpoly;
    ip.N = p->N;
    ip.num_samples = p->num_samples;
    ip.region_size = p->region_size;
    ip.one = p->one_t32;
    ip.max_abs = p->max_abs_coef;
    ip.n_out = n_out;
    ip.n_terms = nnz;
    ip.n_rows = n_in_rows;
    ip.k = k;
    std::vector<uint2> fwd, inv;
    make_twiddles(p->N, &fwd, &inv);
    std::vector<int32_t> bias_v(n_out, 0);
    if (bias) std::memcpy(bias_v.data(), bias, n_out * 4);
    auto fail = [&](idash_status s) {
        idash_model_free(m);
        return s;
    };
    idash_status s = ctx->check_cuda(cudaEventCreateWithFlags(&ip.used, cudaEventDisableTiming), "cudaEventCreate");
    auto up = [&](void **dst, const void *src, size_t bytes, const char *what) {
        if (s != IDASH_OK) return;
        s = ctx->check_cuda(cudaMalloc(dst, std::max<size_t>(bytes, 16)), what);
        if (s == IDASH_OK && bytes) s = ctx->check_cuda(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice), what);
    };
    // groups of outputs that read the same rows in the same order
    ip.group_first.clear();
    std::vector<uint32_t> slot(nnz);
    for (uint64_t o = 0; o < n_out;) {
        uint64_t e = o + 1;
        const uint64_t len = term_ptr[o + 1] - term_ptr[o];
        while (e < n_out && e - o < kGroupMax && term_ptr[e + 1] - term_ptr[e] == len &&
               std::equal(term_feat + term_ptr[o], term_feat + term_ptr[o + 1], term_feat + term_ptr[e]))
            ++e;
        ip.group_first.push_back(o);
        // the group's weights: [term][prime][output]
        for (uint64_t x = o; x < e; ++x)
            for (uint64_t i = 0; i < len; ++i)
                slot[term_ptr[x] + i] = ip_slot(2 * term_ptr[o] + i * 2 * (e - o) + (x - o), uint32_t(e - o));
        o = e;
    }
    ip.group_first.push_back(n_out);
    up(reinterpret_cast<void **>(&ip.d_group_first), ip.group_first.data(), ip.group_first.size() * 8,
       "intpoly groups");
    up(reinterpret_cast<void **>(&ip.d_term_ptr), term_ptr, (n_out + 1) * 8, "intpoly term_ptr");
    up(reinterpret_cast<void **>(&ip.d_term_row), term_feat, nnz * 4, "intpoly term rows");
    up(reinterpret_cast<void **>(&ip.d_slot), slot.data(), nnz * 4, "intpoly slots");
    up(reinterpret_cast<void **>(&ip.d_bias), bias_v.data(), n_out * 4, "intpoly bias");
    up(reinterpret_cast<void **>(&ip.d_tw), fwd.data(), fwd.size() * sizeof(uint2), "intpoly twiddles");
    up(reinterpret_cast<void **>(&ip.d_itw), inv.data(), inv.size() * sizeof(uint2), "intpoly twiddles");
    if (s == IDASH_OK)
        s = ctx->check_cuda(cudaMalloc(&ip.d_w_hat, std::max<size_t>(nnz * 2 * p->N * 4, 16)), "cudaMalloc(W^)");
    if (s != IDASH_OK) return fail(s);
    // Model polynomials -> NTT, through a bounded device staging buffer when on the host.
    const uint64_t chunk = term_poly_on_device ? nnz : std::min<uint64_t>(nnz, (uint64_t(1) << 28) / p->N);
    int16_t *stage = nullptr;
    if (!term_poly_on_device && nnz &&
        (s = ctx->check_cuda(cudaMalloc(&stage, chunk * p->N * 2), "cudaMalloc(model staging)")) != IDASH_OK)
        return fail(s);
    for (uint64_t t0 = 0; t0 < nnz && s == IDASH_OK; t0 += chunk) {
        const uint64_t n = std::min(chunk, nnz - t0);
        const int16_t *src = term_poly + t0 * p->N;
        if (!term_poly_on_device) {
            s = ctx->check_cuda(cudaMemcpy(stage, src, n * p->N * 2, cudaMemcpyHostToDevice), "model upload");
            src = stage;
        }
        if (s != IDASH_OK) break;
        s = ctx->check_cuda(launch_ntt_model(ip, src, t0, n, ctx, ctx->stream), "k_ntt launch");
        if (s == IDASH_OK) s = idash_sync(ctx);
    }
    cudaFree(stage);
    if (s != IDASH_OK) {
        if (s == IDASH_ERR_INDEX) ctx->last_error = "a model coefficient exceeds max_abs_coef";
        return fail(s);
    }
    ctx->models.insert(m);
    *model = m;
    return IDASH_OK;
}

extern "C" idash_status idash_model_intpoly_set_weights(idash_model *m, const int16_t *d_term_poly, void *stream) {
    if (!m) return IDASH_ERR_INVALID_ARGUMENT;
    idash_ctx *ctx = m->ctx;
    if (m->form != Form::kIntPoly || !m->intpoly) return ctx->fail(IDASH_ERR_STATE, "not an integer-polynomial model");
    IntpolyModel &ip = *m->intpoly;
    if (ip.n_terms == 0) return IDASH_OK;
    if (!d_term_poly) return IDASH_ERR_INVALID_ARGUMENT;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    IntpolyTurn turn(ip, st);
    idash_status s = ctx->check_cuda(turn.begin(), "wait for the model's last call");
    if (s == IDASH_OK) s = ctx->check_cuda(launch_ntt_model(ip, d_term_poly, 0, ip.n_terms, ctx, st), "k_ntt launch");
    if (s == IDASH_OK) s = ctx->check_cuda(turn.end(), "record the model's last call");
    return s;
}

extern "C" idash_status idash_score_intpoly_device(idash_model *m, const void *d_in, const idash_row_layout *il,
                                                   uint64_t out_begin, uint64_t out_end, void *d_out,
                                                   const idash_row_layout *ol, void *stream) {
    if (!m || !d_in || !d_out || !il || !ol) return IDASH_ERR_INVALID_ARGUMENT;
    idash_ctx *ctx = m->ctx;
    if (m->form != Form::kIntPoly || !m->intpoly) return ctx->fail(IDASH_ERR_STATE, "not an integer-polynomial model");
    IntpolyModel &ip = *m->intpoly;
    if (out_begin > out_end || out_end > ip.n_out) return ctx->fail(IDASH_ERR_INVALID_ARGUMENT, "bad output range");
    const uint64_t payload = uint64_t(2) * ip.N * 4;
    if (il->row_stride % 16 || ol->row_stride % 16 || il->payload_offset + payload > il->row_stride ||
        ol->payload_offset + payload > ol->row_stride ||
        ((reinterpret_cast<uintptr_t>(d_in) + il->payload_offset) & 15u) ||
        ((reinterpret_cast<uintptr_t>(d_out) + ol->payload_offset) & 15u))
        return ctx->fail(IDASH_ERR_INVALID_ARGUMENT, "row layout: stride or alignment");
    if (out_begin == out_end) return IDASH_OK;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    IntpolyTurn turn(ip, st);
    idash_status s = ctx->check_cuda(turn.begin(), "wait for the model's last call");
    if (s != IDASH_OK) return s;
    if (ip.c_hat_rows < ip.n_rows) {
        if ((s = ctx->check_cuda(cudaStreamSynchronize(st), "sync before growing C^")) != IDASH_OK) return s;
        cudaFree(ip.d_c_hat);
        ip.d_c_hat = nullptr;
        ip.c_hat_rows = 0;
        if ((s = ctx->check_cuda(cudaMalloc(&ip.d_c_hat, std::max<uint64_t>(ip.n_rows, 1) * 4 * ip.N * 4),
                                 "cudaMalloc(C^)")) != IDASH_OK)
            return s;
        ip.c_hat_rows = ip.n_rows;
    }
    if (ip.n_rows) {
        k_ntt<int32_t><<<ntt_grid(4 * ip.n_rows, 2, ctx), kNttThreads, 0, st>>>(
            static_cast<const uint8_t *>(d_in) + il->payload_offset, il->row_stride, 2 * ip.n_rows, ip.d_tw, ip.k, 0,
            nullptr, ip.d_c_hat, ctx->d_err);
        if ((s = ctx->check_cuda(cudaGetLastError(), "k_ntt launch")) != IDASH_OK) return s;
    }
    IntpolyArgs a{};
    a.term_ptr = ip.d_term_ptr;
    a.term_row = ip.d_term_row;
    a.group_first = ip.d_group_first;
    {
        // groups holding outputs of [out_begin, out_end)
        const auto &G = ip.group_first;
        a.group_begin = uint64_t(std::upper_bound(G.begin(), G.end() - 1, out_begin) - G.begin()) - 1;
        a.group_end = uint64_t(std::lower_bound(G.begin(), G.end() - 1, out_end) - G.begin());
    }
    a.w_hat = ip.d_w_hat;
    a.c_hat = ip.d_c_hat;
    a.bias = ip.d_bias;
    a.itw = ip.d_itw;
    a.k = ip.k;
    a.N = ip.N;
    a.num_samples = ip.num_samples;
    a.region_size = ip.region_size;
    a.n_rows = uint32_t(ip.n_rows);
    a.one = ip.one;
    a.out_begin = out_begin;
    a.out_end = out_end;
    a.out = static_cast<uint8_t *>(d_out) + ol->payload_offset;
    a.out_stride = ol->row_stride;
    a.err = ctx->d_err;
    // the ring needs more than the default 48 KiB of dynamic shared memory
    if ((s = ctx->check_cuda(cudaFuncSetAttribute(k_intpoly_score, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  int(kIpScoreSmem)),
                             "k_intpoly_score shared memory")) != IDASH_OK)
        return s;
    const uint32_t grid = uint32_t(std::min<uint64_t>(a.group_end - a.group_begin, ctx->sm_count));
    k_intpoly_score<<<grid, kScoreBlock, kIpScoreSmem, st>>>(a);
    s = ctx->check_cuda(cudaGetLastError(), "k_intpoly_score launch");
    if (s == IDASH_OK) s = ctx->check_cuda(turn.end(), "record the model's last call");
    if (s == IDASH_OK) ctx->stats.kernel_launches += 2;
    return s;
}

extern "C" idash_status idash_synth_int16_device(idash_ctx *ctx, uint64_t seed, uint64_t n, int32_t max_abs,
                                                 int16_t *d_out, void *stream) {
    if (!ctx || !d_out || max_abs <= 0 || max_abs > 16383) return IDASH_ERR_INVALID_ARGUMENT;
    if (n == 0) return IDASH_OK;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    const uint32_t grid = uint32_t(std::min<uint64_t>((n + 255) / 256, uint64_t(ctx->sm_count) * 16));
    k_synth_int16<<<grid, 256, 0, st>>>(seed, n, max_abs, d_out);
    return ctx->check_cuda(cudaGetLastError(), "k_synth_int16 launch");
}
