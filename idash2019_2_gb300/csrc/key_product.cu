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
// Layout.  M = 128 of an MMA is 32 rows x 3 digits (quadrant w of the TMEM
// lanes: digit d of row 8 w + r in lane 32 w + 8 d + r; eight lanes of each
// quadrant stay zero), so that a thread's part of a 16-lane TMEM load holds
// the same row's digits: with 40 rows on 120 lanes the digits had to be
// exchanged between lanes, and that bound the kernel.  N = up to 256
// coefficients j.  T is Toeplitz and an 8 x 8 core matrix of it depends only
// on the difference of its group indices, so with the k-groups in reverse
// order the whole of T is a table of 2N/8 - 1 core matrices (32 KB at
// N = 1024) that the descriptor walks with both strides 128 bytes: it is
// built once per CTA from the key bits and never reloaded.
//
// Structure: one CTA of 18 warps per SM, persistent over items (32 rows, a
// pair of column tiles t0, t1).
//   warps 10-17 in two teams that take chunks in turn: load 64-word pieces of
//              the rows (two ahead, in registers), split them into digits,
//              store them as the MMA's A (k-groups 16 bytes off a multiple of
//              128 apart, so that the eight groups of a row, one per lane, are
//              in different banks);
//   warps 8, 9 issue the MMAs of t0 and t1 (one warp for both took 628 cycles
//              per chunk and tile, of which the MMAs are 516).  The epilogues
//              come in turn, so that one tile's runs under the other's MMAs
//              although the two accumulators (2 x 256 columns) fill TMEM;
//   warps 0-7  epilogue of t0 and t1 in turn: each lane joins the digit sums of
//              two consecutive coefficients of a row and finishes them; the
//              row's body words are in registers before the sums are ready.
// Every wait is bounded and ends when another role raised the abort flag.
//
// What bounds it: 242,646 masks x 1,000 coefficients take 0.96 ms (6.90 ms as
// sums over the key's set bits on CUDA cores; 1.64 ms with 40 rows a tile, the
// digits exchanged by shuffles and one warp for both tiles' MMAs).  An item
// (32 rows x 512 coefficients) takes 18,000 cycles, of which its MMAs are
// 16,500 (0.83 ms); reading and writing 3.0 GB would take 0.45 ms.
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

constexpr uint32_t kRows = 32;        // rows per item
constexpr uint32_t kChunkWords = 64;  // mask words per pipeline chunk (four K = 16 steps)
constexpr uint32_t kMaxStages = 10;
// chunks of A in shared memory, beside the table
__host__ __device__ constexpr uint32_t kp_stages(uint32_t N) { return N <= 1024 ? kMaxStages : 8; }
constexpr uint32_t kGroupBytes = 128 * 16 + 16;  // one k-group (8 words) of A: 16 core matrices and the padding
constexpr uint32_t kStageBytes = (kChunkWords / 8) * kGroupBytes;
constexpr uint32_t kTileMax = 256;    // columns of one accumulator
constexpr uint32_t kEpiWarps = 8;     // two per quadrant, half of a tile's columns each
constexpr uint32_t kMmaWarp = kEpiWarps, kConvWarp0 = kMmaWarp + 2;
constexpr uint32_t kConvTeams = 2, kTeamWarps = 4;  // the stages are a multiple of the teams
constexpr uint32_t kConvWarps = kConvTeams * kTeamWarps;
constexpr uint32_t kKpThreads = 32 * (kConvWarp0 + kConvWarps);
constexpr uint32_t kHeader = 1024;
constexpr uint32_t kMagicBits = 0x3F400000u;  // 0.75f
static_assert(kRows * (kChunkWords / 8) == 2 * 32 * kTeamWarps, "two 8-word units per converter thread and chunk");

struct KpShared {
    uint64_t a_full[kMaxStages], a_empty[kMaxStages];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t drain;
    uint32_t tmem_base, abort;
    uint32_t key[kKeyMaxN / 32];
};
static_assert(sizeof(KpShared) <= kHeader, "header area");

__host__ __device__ constexpr uint32_t kp_table_bytes(uint32_t N) { return (2 * N / 8) * 128; }
// at least 120 KB, so that no second CTA (which would wait for this one's
// tensor memory) fits on the SM
constexpr size_t kp_smem(uint32_t N) { return kHeader + kp_table_bytes(N) + size_t(kp_stages(N)) * kStageBytes; }
static_assert(kp_smem(32) > 120 * 1024, "one CTA per SM");
static_assert(kp_smem(1024) <= 227 * 1024 && kp_smem(kKeyMaxN) <= 227 * 1024, "shared memory");

__device__ __forceinline__ const uint8_t *kp_row(const KeyProductArgs &a, uint64_t r) {
    return a.rows + (a.row_map ? uint64_t(a.row_map[r]) : r) * a.stride;
}

// 8 words from p: 16-byte loads when the rows allow them.
__device__ __forceinline__ void kp_load(const uint32_t *p, bool vec, uint32_t (&v)[8]) {
    if (vec) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 q = reinterpret_cast<const uint4 *>(p)[i];
            v[4 * i] = q.x;
            v[4 * i + 1] = q.y;
            v[4 * i + 2] = q.z;
            v[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i];
    }
}

// 32 columns of 16 TMEM lanes: of columns 8 k + 2 (lane % 4) and the next,
// r[4 k] and r[4 k + 1] in TMEM lane lane / 4, r[4 k + 2] and r[4 k + 3] eight
// lanes on.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}

// A digit sum's accumulator as an integer plus kMagicBits.
__device__ __forceinline__ uint32_t kp_digit(uint32_t acc) {
    return __float_as_uint(__fadd_rn(__uint_as_float(acc), 0.75f));
}

// T's entry at difference d = j - k as fp16 bits.
__device__ __forceinline__ uint32_t kp_entry(const uint32_t *key, uint32_t N, int32_t d) {
    const uint32_t i = d >= 0 ? uint32_t(d) : uint32_t(int32_t(N) + d);
    if (i >= N || !((key[i / 32] >> (i % 32)) & 1u)) return 0u;
    return d >= 0 ? 0x3C00u : 0xBC00u;  // 1 or -1
}

// kScores: decryption (scores from b - a*s), else b += a*s.
// kHalf: N = 32, one chunk of which the first half is the row's words (told apart
// at run time, the issuing loop made 1,000 coefficients 3% slower).
template <bool kScores, bool kHalf>
__global__ void __launch_bounds__(kKpThreads, 1) k_key_product(const __grid_constant__ KeyProductArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    KpShared &sh = *reinterpret_cast<KpShared *>(smem);
    uint8_t *table = smem + kHeader;
    uint8_t *stages = table + kp_table_bytes(a.N);
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t N = a.N, groups = N / 8, n_chunks = kHalf ? 1 : N / kChunkWords;
    const uint32_t n_stages = kp_stages(N);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < n_stages; ++s) {
            mbar_init(&sh.a_full[s], kTeamWarps);
            mbar_init(&sh.a_empty[s], 2);
        }
        for (uint32_t t = 0; t < 2; ++t) {
            mbar_init(&sh.acc_full[t], 1);
            mbar_init(&sh.acc_empty[t], kEpiWarps);
        }
        mbar_init(&sh.drain, 2);
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
    // the eight lanes of each quadrant without a digit stay zero
    for (uint32_t x = threadIdx.x; x < n_stages * (kChunkWords / 8) * 32; x += kKpThreads) {
        const uint32_t m = 32 * (x / 8 % 4) + 24 + x % 8;
        sts_v4(smem_addr(stages + (x / 32) * kGroupBytes + m * 16), 0, 0, 0, 0);
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
        // Team `team` takes chunks team, team + 2, ... of the CTA's stream.
        const uint32_t team = (warp - kConvWarp0) / kTeamWarps;
        const uint32_t cid = threadIdx.x - 32 * (kConvWarp0 + team * kTeamWarps);
        const uint32_t l = cid % 8, row = cid / 8;  // group l of each chunk, rows `row` and `row + 16`
        const uint64_t total = my_items * n_chunks;
        uint64_t f_item = blockIdx.x;  // the next load's item and chunk
        uint32_t f_c = team;
        const uint32_t *f_src[2];
        auto open = [&]() {
            for (; f_c >= n_chunks; f_c -= n_chunks) f_item += gridDim.x;
            const uint64_t r0 = (f_item / a.pairs) * kRows + row;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint64_t r = r0 + h * (kRows / 2);
                f_src[h] = f_item < a.items && r < a.n_rows && (!kHalf || l < groups)
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
                    kp_load(f_src[h] - kChunkWords * f_c, a.vec_rows, v[h]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[h][e] = 0;
                }
            }
            f_c += kConvTeams;
            if (f_c >= n_chunks) open();
        };
        open();
        uint32_t buf[2][2][8];
        fetch(buf[0]);
        fetch(buf[1]);
        const uint32_t at = smem_addr(stages) + l * kGroupBytes + (32 * (row / 8) + row % 8) * 16;
        uint32_t s = team, round = 0;
        auto step = [&](uint32_t (&v)[2][8]) {
            if (round > 0 && !tc_warp_wait(&sh.abort, &sh.a_empty[s], (round - 1) & 1u, a.err, lane)) return false;
            const uint32_t dst = at + s * kStageBytes;
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
                // 16 rows on: two quadrants
#pragma unroll
                for (uint32_t d = 0; d < 3; ++d)
                    sts_v4(dst + (64 * h + 8 * d) * 16, u[d][0], u[d][1], u[d][2], u[d][3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.a_full[s]);
            s += kConvTeams;
            if (s >= n_stages) {
                s -= n_stages;
                ++round;
            }
            fetch(v);
            return true;
        };
        bool ok = true;
        for (uint64_t g = team; ok && g < total; g += 2 * kConvTeams) {
            ok = step(buf[0]);
            if (ok && g + kConvTeams < total) ok = step(buf[1]);
        }
    } else if (warp >= kMmaWarp) {
        // ----------------------------------------------------------------- MMA
        // Each lane leaves by its own verdict: nothing in the loop waits for the
        // other lanes.
        const bool leader = elect_one();
        const uint32_t t = warp - kMmaWarp, d = tmem + t * kTileMax;
        const uint64_t a_desc = umma_desc(smem_addr(stages), kGroupBytes, 128);
        const uint64_t t_desc = umma_desc(smem_addr(table), 128, 128);
        uint32_t s = 0, parity = 0;
        uint64_t item = blockIdx.x;
        bool ok = true;
        for (uint32_t i = 0; ok && i < my_items; ++i, item += gridDim.x) {
            uint32_t n0, w;
            tile_of(item, t, n0, w);
            const uint32_t idesc = umma_idesc_f16(128, w);
            uint64_t b = t_desc + n0;  // n0 / 8 core matrices of 128 bytes, in 16-byte units
            if (i > 0 && !(ok = tc_wait(&sh.abort, &sh.acc_empty[t], (i - 1) & 1u, a.err))) break;
            tc_fence_after();
            for (uint32_t c = 0; c < n_chunks; ++c) {
                if (!(ok = tc_wait(&sh.abort, &sh.a_full[s], parity, a.err))) break;
                tc_fence_after();
                const uint64_t da = a_desc + s * (kStageBytes / 16);
                if (leader) {
                    if (w) {
#pragma unroll
                        for (uint32_t j = 0; j < (kHalf ? 2 : kChunkWords / 16); ++j)
                            umma_f16(d, da + j * (2 * kGroupBytes / 16), b + j * 16, idesc, c + j > 0 ? 1u : 0u);
                    }
                    umma_commit(&sh.a_empty[s]);
                    if (c + 1 == n_chunks) umma_commit(&sh.acc_full[t]);
                }
                b += (kChunkWords / 8) * (128 / 16);
                if (++s == n_stages) {
                    s = 0;
                    parity ^= 1u;
                }
            }
        }
        // every MMA issued has completed before TMEM is released
        if (leader) umma_commit(&sh.drain);
        mbar_wait_bounded(&sh.drain, 0, nullptr);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        constexpr uint32_t kMagicSum = kMagicBits + (kMagicBits << 11) + (kMagicBits << 22);
        const uint32_t half = warp / 4, quadrant = warp % 4, c_lane = 2 * (lane % 4);
        uint64_t it = 0;
        for (; it < 2 * my_items; ++it) {
            const uint64_t i = it / 2, item = blockIdx.x + i * gridDim.x;
            const uint32_t t = it % 2;
            const uint64_t row = (item / a.pairs) * kRows + 8 * quadrant + lane / 4;
            uint32_t n0, w;
            tile_of(item, t, n0, w);
            // this warp's columns [first, last) of the tile, a lane's 8 k + c_lane
            // and the next of every 32
            const uint32_t middle = (w / 2 + 15u) & ~15u;
            const uint32_t first = half ? middle : 0u, last = half ? w : middle;
            const bool has = row < a.n_rows;
            uint32_t *body = nullptr;
            if (has) body = reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(kp_row(a, row))) + N + n0;
            uint32_t *dst = kScores ? reinterpret_cast<uint32_t *>(a.scores) + row * a.n_coef + n0 : body;
            const uint32_t n_has = has ? min(last, a.n_coef - min(a.n_coef, n0)) : 0u;  // live columns end here
            uint2 b[kTileMax / 64][4];
#pragma unroll
            for (uint32_t g = 0; g < kTileMax / 64; ++g)
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t c = first + 32 * g + 8 * k + c_lane;
                    if (c >= n_has) continue;
                    if (a.vec_rows) b[g][k] = *reinterpret_cast<const uint2 *>(body + c);
                    else b[g][k] = make_uint2(body[c], body[c + 1]);  // inside the row: N is even
                }
            if (!tc_warp_wait(&sh.abort, &sh.acc_full[t], uint32_t(i) & 1u, a.err, lane)) break;
            tc_fence_after();
            const uint32_t base = tmem + ((32 * quadrant) << 16) + t * kTileMax + first;
#pragma unroll
            for (uint32_t g = 0; g < kTileMax / 64; ++g) {
                if (first + 32 * g >= last) break;
                uint32_t lo[16], hi[16];  // digits 0 and 1, digit 2 and the zero lanes
                tmem_ld_16x32(base + 32 * g, lo);  // past `last`: columns of this accumulator, not used
                tmem_ld_16x32(base + 32 * g + (16u << 16), hi);
                tmem_wait_ld();
                if (first + 32 * (g + 1) >= last) {  // the sums are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.acc_empty[t]);
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    uint32_t v[2] = {b[g][k].x, b[g][k].y};
#pragma unroll
                    for (uint32_t e = 0; e < 2; ++e) {
                        const uint32_t p = kp_digit(lo[4 * k + e]) + (kp_digit(lo[4 * k + 2 + e]) << 11) +
                                           (kp_digit(hi[4 * k + e]) << 22) - kMagicSum;
                        if (kScores)
                            v[e] = __float_as_uint(__int2float_rn(int32_t(v[e] - p)) * 0x1p-32f);
                        else
                            v[e] += p;
                    }
                    const uint32_t c = first + 32 * g + 8 * k + c_lane;
                    if (c + 2 <= n_has && (kScores ? a.vec_scores : a.vec_rows)) {
                        *reinterpret_cast<uint2 *>(dst + c) = make_uint2(v[0], v[1]);
                    } else {
                        if (c < n_has) dst[c] = v[0];
                        if (c + 1 < n_has) dst[c + 1] = v[1];
                    }
                }
            }
            if (first >= last && lane == 0) mbar_arrive(&sh.acc_empty[t]);
        }
        // given up: no body stays without its product
        for (; !kScores && it < 2 * my_items; ++it) {
            const uint64_t item = blockIdx.x + (it / 2) * gridDim.x;
            const uint64_t row = (item / a.pairs) * kRows + 8 * quadrant + lane / 4;
            uint32_t n0, w;
            tile_of(item, it % 2, n0, w);
            if (row >= a.n_rows) continue;
            uint32_t *body = reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(kp_row(a, row))) + N;
            const uint32_t middle = (w / 2 + 15u) & ~15u, end = min(n0 + (half ? w : middle), a.n_coef);
            for (uint32_t j = n0 + (half ? middle : 0u) + lane % 4; j < end; j += 4) body[j] = 0;
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem, 2 * kTileMax);
}

// The bodies' coefficients [0, n_coef) to zero, a CTA to a row in turn.
__global__ void k_clear_bodies(const __grid_constant__ KeyProductArgs a) {
    for (uint64_t r = blockIdx.x; r < a.n_rows; r += gridDim.x) {
        uint32_t *body = reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(kp_row(a, r))) + a.N;
        for (uint32_t j = threadIdx.x; j < a.n_coef; j += blockDim.x) body[j] = 0;
    }
}

}  // namespace

cudaError_t launch_key_product(KeyProductArgs a, int sm_count, cudaStream_t s) {
    if (a.n_rows == 0 || a.n_coef == 0) return cudaSuccess;
    if (!key_product_supported(a.N) || (a.N & (a.N - 1)) || a.n_coef > a.N) return cudaErrorInvalidValue;
    const uint64_t row_tiles = (a.n_rows + kRows - 1) / kRows;
    const uint32_t coef_pad = (a.n_coef + 15u) & ~15u;
    // Pairs of column tiles per 32 rows: as few as the accumulators allow (a
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
    a.vec_scores = ((reinterpret_cast<uintptr_t>(a.scores) | (uint64_t(a.n_coef) * 4)) & 7u) == 0;
    const bool half = a.N < kChunkWords;
    auto *fn = a.scores ? (half ? k_key_product<true, true> : k_key_product<true, false>)
                        : (half ? k_key_product<false, true> : k_key_product<false, false>);
    fn<<<uint32_t(std::min<uint64_t>(a.items, uint64_t(sm_count))), kKpThreads, kp_smem(a.N), s>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess && !a.scores)
        k_clear_bodies<<<uint32_t(std::min<uint64_t>(a.n_rows, uint64_t(sm_count) * 8)), 256, 0, s>>>(a);
    return e;
}

cudaError_t configure_key_product() {
    for (auto *fn : {k_key_product<true, false>, k_key_product<false, false>, k_key_product<true, true>,
                     k_key_product<false, true>}) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   int(std::max(kp_smem(1024), kp_smem(kKeyMaxN))));
        if (e != cudaSuccess) return e;
    }
    cudaFuncAttributes loaded{};  // now, not when something else has failed
    return cudaFuncGetAttributes(&loaded, k_clear_bodies);
}

}  // namespace idash
