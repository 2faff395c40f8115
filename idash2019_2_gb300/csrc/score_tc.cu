// Scoring on the tensor cores: out_o = bias_o + sum_k coef[o][k] * row_k, per
// column, in Z/2^32 - the accumulate of cloud_compute_score
// (tLweAddMulTo per term, eval/idash.cpp:800-819) as a dense product
//   D[outputs x columns] = A[outputs x rows] * B[rows x columns]
// per block of up to 128 consecutive outputs, on tcgen05.mma.
//
// Exactness.  The operands are small integers held exactly in fp16 and
// summed exactly in fp32: an error-free splitting of an integer product into
// digit products, as in the published tensor-core methods that emulate exact
// or high-precision matrix products by splitting (Mukunoki, Ozaki, Ogita and
// Imamura, "DGEMM using Tensor Cores, and Its Accurate and Reproducible
// Versions", ISC 2020).  A ciphertext word is its four bytes x = sum_i b_i
// 256^i; the fp16 bit pattern of a byte (a subnormal) is the value b * 2^-24,
// so a byte is its own encoding.  A coefficient is c0 + 256 c1, c0 in [-128,
// 127].  Digit products land in four accumulators by shift: D_s = sum over
// i + j = s of A_j * B_i, s = 0..3, and out = sum_s 256^s D_s (mod 2^32).
// The planner bounds K so that with balanced digits b - 128 every partial sum
// stays below 2^22 units of 2^-24 (plan.hpp), so with b in [0, 255] below
// 2^23, which fp32 holds exactly.  The epilogue adds 0.75 - 128 S_s 2^-24
// (S_s: the output's digit sum that multiplies D_s): the result is 0.75 plus
// the balanced sum, in [0.5, 1), where the last place is 2^-24 and the bits
// are an integer; the plan's per-output constant puts 128 S_s back.
//
// Structure (one persistent CTA per SM over work units of (block, run of
// 64-column slices)).  A role's hand-offs and lookups take hundreds of
// cycles, as long as the work itself on a tile, so the roles that would bound
// the kernel come in teams that take tiles or chunks in turn:
//   producers   (one or two warps) per chunk of 32 rows, the rows' 64-column
//               slices: one 2D tensor copy when the chunk's rows are
//               consecutive, else 16-byte copies, two rows per instruction;
//   digits      (one warp) loads the block's coefficient digits (one bulk
//               copy, kept in shared memory for the unit, the next unit's
//               beside them where they fit);
//   converters  (two teams of two warps or three of four) eight rows of a
//               column -> one 16-byte row of each of the four byte planes, in
//               the MMA's no-swizzle K-major layout with the planes side by
//               side along N;
//   MMA         (one warp) owns the 512 TMEM columns and issues two
//               tcgen05.mma per K = 16 step (M = 128: c0 times the four
//               planes, N = 256, and c1 times the first three, N = 192, one
//               accumulator to the right) into a double-buffered set of four
//               fp32 accumulators;
//   epilogue    (one or two teams of eight warps) tcgen05.ld of the
//               accumulators (a warp reads 32 TMEM lanes, one output each,
//               and half the columns), the digit recombination, bias and
//               zeroed columns, staged in shared memory (128-byte swizzle)
//               and stored by 2D tensor copies of 32 rows x 32 columns, or
//               row by row where the 32 rows are not all wanted or not
//               consecutive.
// Several regions to a row (kRotated): a slot is a row times X^(-m), so the
// producers (six warps) copy a slot's columns from m on, round the
// polynomial's end, in the largest pieces that stay aligned, and the
// converters negate those that went round.  The slices past the last region's
// columns are zeros: the digits' warp stores them from a box of zeros, and
// they cost the other roles nothing.
// What bounds it, and what it measured: 5 neighbours (K = 64, 2.4 GB) the
// roles' instructions, about 5200 a tile: 0.41 ms against 0.36 ms of memory
// traffic; 30 neighbours (K = 192) the conversion and the MMAs, 448 cycles of
// MMA per 32 rows.
// Every wait is bounded; a wait that expires records IDASH_ERR_DEVICE_TIMEOUT,
// raises a CTA-wide abort flag that ends the other roles' waits, and each
// role then waits (bounded) for its own copies and MMAs in flight before the
// TMEM columns are freed.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "score_kernels.cuh"
#include "tcgen05.cuh"

namespace idash {

namespace {

constexpr uint32_t kN = kTcSliceWords;  // 64 columns per tile
constexpr uint32_t kM = kTcRows;        // 128 outputs per block
constexpr uint32_t kChunk = 32;         // rows per pipeline chunk (two MMA K-steps)
constexpr uint32_t kMaxChunks = kTcMaxK / kChunk;
constexpr uint32_t kAccStages = 2;
constexpr uint32_t kTcRotStages = 6;  // raw stages where rows are rotated
constexpr uint32_t kMaxAStages = 2, kMaxRawStages = 8, kMaxDigStages = 4;
constexpr uint32_t kRawStageBytes = kChunk * kN * 4;
constexpr uint32_t kGroupBytes = 4 * kN * 16;           // 8 rows of the four planes
constexpr uint32_t kDigStageBytes = (kChunk / 8) * kGroupBytes;
constexpr uint32_t kOutBox = 32 * 32 * 4;               // one stored box: 32 rows x 32 columns
constexpr uint32_t kHeader = 2048;
constexpr uint32_t kZeroBox = 12 * 1024, kRotHeader = kZeroBox + kOutBox;  // with TcRot and a box of zeros
// Warps: kEpi teams of eight (one, or one per accumulator stage), kProducers
// producers, one each of MMA and digit loads, then kConv converter teams of
// kConvWarps.  A parity tells only two successive phases of a barrier apart,
// so a team must meet all phases of the stages it waits for in turn: a stage
// belongs to one team.
constexpr uint32_t kEpiWarps = 8;
constexpr uint32_t tc_threads(uint32_t epi, uint32_t conv, uint32_t conv_warps, uint32_t producers) {
    return 32 * (kEpiWarps * epi + producers + 2 + conv_warps * conv);
}
constexpr uint32_t kTmemCols = 512;                     // 2 stages x 4 accumulators x 64 columns
constexpr uint32_t kIdescAll = umma_idesc_f16(kM, 4 * kN), kIdescHigh = umma_idesc_f16(kM, 3 * kN);
constexpr uint32_t kMagic = 0x3F400000u;                // bits of 0.75
constexpr uint32_t kMagicSum = kMagic + (kMagic << 8) + (kMagic << 16) + (kMagic << 24);
// one CTA per SM, so the CTA owns all of TMEM
constexpr size_t kMinSmem = 120 * 1024;
constexpr size_t kMaxSmem = 227 * 1024;

// Teams and buffers for a plan whose largest padded K is k: the first that
// fits.  Small K: the epilogue is most of the work (two teams, one per
// accumulator stage) and copies in flight cover the memory's latency (eight
// raw stages up to K = 64, six up to 80).  Large K: the conversion is (three
// teams of four warps).  42,000 outputs over 2,100 rows, first and second
// kind: K = 48 0.101 and 0.117 ms, K = 80 0.114 and 0.123, K = 96 0.126 and
// 0.122; 6,000 outputs, K = 128 to 160: 0.076 to 0.090 and 0.071 to 0.081.
// Raw and digit stages are multiples of the converter teams (see above), raw
// stages of the producers too.
struct TcShape {
    uint32_t epi, conv, conv_warps;
    uint32_t a_stages;    // blocks' coefficient digits
    uint32_t dig_stages;  // chunks of byte planes
    uint32_t raw_stages;  // chunks of ciphertext words
    constexpr size_t smem(uint32_t k, bool rotated) const {
        const size_t n = (rotated ? kRotHeader : kHeader) + a_stages * size_t(tc_a_bytes(k)) +
                         dig_stages * size_t(kDigStageBytes) + raw_stages * size_t(kRawStageBytes) + kEpiWarps * epi * size_t(kOutBox);
        return n < kMinSmem ? kMinSmem : n;
    }
};
constexpr TcShape kTcShapes[] = {{2, 2, 2, 2, 2, 8}, {2, 2, 2, 2, 2, 6}, {1, 3, 4, 2, 3, 6}, {1, 3, 4, 1, 3, 6}};
// Rotated rows: the producers are most of the work.
constexpr TcShape kTcRotShapes[] = {{1, 2, 4, 2, 2, 6}, {1, 2, 4, 1, 2, 6}};
static_assert(kTcShapes[3].smem(kTcMaxK, false) <= kMaxSmem && kTcRotShapes[1].smem(kTcMaxK, true) <= kMaxSmem, "K");
const TcShape *tc_shape(uint32_t k, bool rotated) {
    if (rotated) {
        for (const TcShape &x : kTcRotShapes)
            if (x.smem(k, true) <= kMaxSmem) return &x;
        return nullptr;
    }
    for (const TcShape &x : kTcShapes)
        if (x.smem(k, false) <= kMaxSmem) return &x;
    return nullptr;
}

struct TcBars {
    uint64_t a_full[kMaxAStages], a_empty[kMaxAStages], drain;
    uint64_t raw_full[kMaxRawStages], raw_empty[kMaxRawStages];
    uint64_t dig_full[kMaxDigStages], dig_empty[kMaxDigStages];
    uint64_t acc_full[kAccStages], acc_empty[kAccStages];
    uint32_t tmem_base;
    uint32_t abort;
    uint32_t rows[kTcMaxProducers][kTcMaxK];  // the unit's input rows, per producer
};
static_assert(sizeof(TcBars) <= kHeader, "header area");

// Plans with rotated slots: the unit's input rows and rotations, per producer;
// and per raw stage, slot i's columns from[i] .. 63 are to be negated (they
// went round the polynomial's end), if any slot's are.
struct TcRot {
    uint32_t rows[kTcRotProducers][kTcMaxK], rots[kTcRotProducers][kTcMaxK];
    uint32_t from[kTcRotStages][kChunk];
    uint32_t any[kTcRotStages];
};
static_assert(kHeader + sizeof(TcRot) <= kZeroBox, "header area");

// A position in a ring of n stages; parity of the round.
struct Ring {
    uint32_t s = 0, round = 0;
    __device__ __forceinline__ void next(uint32_t n) {
        if (++s == n) {
            s = 0;
            ++round;
        }
    }
};

// A 16-byte shared load that stays before the barrier that follows it.
__device__ __forceinline__ uint4 lds_v4_ordered(uint32_t addr) {
    uint4 v;
    asm volatile("ld.volatile.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr)
                 : "memory");
}

// x + m and y + m as floats, each rounded to nearest, in one instruction.
__device__ __forceinline__ void add2(uint32_t &x, uint32_t &y, float m) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\t"
        "add.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+r"(x), "+r"(y)
        : "f"(m));
}

// 2D tensor copy of the box at (x = column, y = row) into shared memory,
// completed on `bar` as transaction bytes.  x * 4 is a multiple of 16.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int32_t x, int32_t y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// 16 bytes global -> shared (zeros when `bytes` is 0), counted by the
// cp_async_arrive that follows it.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// `bar`'s phase also waits for this thread's cp.async so far.
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.shared.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int32_t x, int32_t y, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x),
                 "r"(y), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// At most kLeft of this thread's store groups still read shared memory.
template <int kLeft>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kLeft) : "memory");
}
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// The CTA's work units blockIdx.x, + gridDim.x, ...: unit u is slices [s0, s1)
// of block `block`.  Stepped without a division.
struct Units {
    uint32_t u, block, part;
    __device__ __forceinline__ explicit Units(const ScoreArgs &a)
        : u(blockIdx.x), block(blockIdx.x / a.units_per_block), part(blockIdx.x % a.units_per_block) {}
    __device__ __forceinline__ bool valid(const ScoreArgs &a) const { return u < a.n_units; }
    __device__ __forceinline__ void next(const ScoreArgs &a) {
        u += gridDim.x;
        block += a.unit_step_blocks;
        part += a.unit_step_parts;
        if (part >= a.units_per_block) {
            part -= a.units_per_block;
            ++block;
        }
    }
    __device__ __forceinline__ uint32_t s0(const ScoreArgs &a) const { return part * a.unit_slices; }
    __device__ __forceinline__ uint32_t s1(const ScoreArgs &a) const {
        return min((part + 1) * a.unit_slices, a.n_slices);
    }
    // the unit's share of the slices that are zeros
    __device__ __forceinline__ uint32_t z0(const ScoreArgs &a) const {
        return a.n_slices + min(part * a.zero_per_unit, a.zero_slices);
    }
    __device__ __forceinline__ uint32_t z1(const ScoreArgs &a) const {
        return a.n_slices + min((part + 1) * a.zero_per_unit, a.zero_slices);
    }
    __device__ __forceinline__ const PlanBlock *header(const ScoreArgs &a) const {
        return a.blocks + a.block_lo + block;
    }
};

// Padded K of the CTA's units, each read one unit ahead of its use.
struct UnitDepths {
    Units ahead;
    uint32_t pending;
    __device__ __forceinline__ explicit UnitDepths(const ScoreArgs &a) : ahead(a), pending(0) { fetch(a); }
    __device__ __forceinline__ void fetch(const ScoreArgs &a) {
        if (ahead.valid(a)) pending = ahead.header(a)->n_groups;
    }
    __device__ __forceinline__ uint32_t next(const ScoreArgs &a) {
        const uint32_t k = pending;
        ahead.next(a);
        fetch(a);
        return k;
    }
};

// Bit i: column c0 + i is in [lo, hi), i < 32.
__device__ __forceinline__ uint32_t columns_in(uint32_t c0, uint32_t lo, uint32_t hi) {
    const uint32_t from = lo > c0 ? min(lo - c0, 32u) : 0u, to = hi > c0 ? min(hi - c0, 32u) : 0u;
    return from < to ? (0xFFFFFFFFu >> (32u - (to - from))) << from : 0u;
}

// The launch's tensor maps: rows (boxes of 64 columns x 32 rows) and outputs
// (32 x 32, 128-byte swizzle).
struct TcMaps {
    CUtensorMap rows, out;
};

// n rows of a chunk that one box does not hold into a raw stage, two rows per
// instruction.  The whole warp calls it.  (Four-row tensor gathers took 270
// cycles each: 10 neighbours over permuted rows 0.324 ms with them, 0.309 ms
// this way.)
__device__ __forceinline__ void load_rows(const ScoreArgs &a, const uint32_t *rows, uint32_t n, uint32_t c0,
                                          uint32_t dst, uint64_t *full, uint32_t lane) {
    const uint32_t half = lane / 16, word = c0 + 4 * (lane % 16);
    const uint32_t bytes = word < a.row_words ? 16u : 0u;  // rows are whole 16-byte pieces apart
    const uint8_t *src = a.in + uint64_t(bytes ? word : 0u) * 4;
    dst += half * (kN * 4) + (lane % 16) * 16;
#pragma unroll 4
    for (uint32_t i = 0; i < n; i += 2)
        cp_async16(dst + i * (kN * 4), src + uint64_t(rows[min(i + half, n - 1)]) * a.in_stride, bytes);
    cp_async_arrive(full);
    __syncwarp();
    if (lane == 0) mbar_arrive(full);
}

template <uint32_t kBytes>
__device__ __forceinline__ void cp_async_words(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(kBytes) : "memory");
}

// (8,000 tags, 24,000 targets, 10 regions to a row: 5 neighbours 0.139 ms, 0.294
// as sums on CUDA cores, 0.091 the memory traffic alone; 20 neighbours 0.183
// and 1.123 ms.  Two producers, and the zeros staged by the epilogue: 0.243 and
// 0.334; six: 0.180 and 0.215.  3 regions, copied word by word: 0.191, 0.323.)
//
// Columns [c0, c0 + 64) of n rotated slots into a raw stage: column j of a
// polynomial of slot X^(-m) * row is the row's word (j + m) mod N, negated
// where j + m >= N (the converters do that).  kBytes divides every rotation.
// The whole warp calls it.
template <uint32_t kBytes>
__device__ __forceinline__ void load_rotated(const ScoreArgs &a, const uint32_t *rows, const uint32_t *rots, uint32_t n,
                                             uint32_t c0, uint32_t dst, uint32_t lane) {
    constexpr uint32_t kWords = kBytes / 4, kLanes = kN / kWords;  // lanes of a slot's 64 words
    const uint32_t mask = a.N - 1, poly = c0 & ~mask, word = lane * kWords % kN;
    const uint32_t j = (c0 & mask) + word;
    const uint8_t *base = a.in + uint64_t(poly) * 4;
    dst += lane * kBytes;  // lanes past a slot's are at the next one's
    if (kLanes <= 32) {
        constexpr uint32_t kSlots = kLanes <= 32 ? 32 / kLanes : 1;
#pragma unroll 4
        for (uint32_t i = 0; i < n; i += kSlots) {
            const uint32_t s = min(i + lane / kLanes, n - 1);
            const uint8_t *src = base + uint64_t(rows[s]) * a.in_stride + ((j + rots[s]) & mask) * 4;
            cp_async_words<kBytes>(dst + i * (kN * 4), src);
        }
    } else {
#pragma unroll 4
        for (uint32_t i = 0; i < n; ++i) {
            const uint8_t *row = base + uint64_t(rows[i]) * a.in_stride;
            const uint32_t t = j + rots[i];
            cp_async_words<kBytes>(dst + i * (kN * 4), row + (t & mask) * 4);
            cp_async_words<kBytes>(dst + i * (kN * 4) + 128, row + ((t + 32) & mask) * 4);
        }
    }
}

// kRotated: rows come rotated (several regions to a row), by kTcRotProducers warps.
template <uint32_t kEpi, uint32_t kConv, uint32_t kConvWarps, uint32_t kProducers, bool kRotated = false>
__global__ void __launch_bounds__(tc_threads(kEpi, kConv, kConvWarps, kProducers), 1)
    k_score_tc(const __grid_constant__ ScoreArgs a, const __grid_constant__ TcMaps maps) {
    constexpr uint32_t kProducerWarp = kEpiWarps * kEpi, kMmaWarp = kProducerWarp + kProducers;
    constexpr uint32_t kDigitWarp = kMmaWarp + 1;
    constexpr uint32_t kConvWarp0 = kDigitWarp + 1;
    extern __shared__ __align__(1024) uint8_t smem[];
    TcBars &sh = *reinterpret_cast<TcBars *>(smem);
    TcRot &rot = *reinterpret_cast<TcRot *>(smem + kHeader);  // kRotated
    uint8_t *stage_out = smem + (kRotated ? kRotHeader : kHeader);
    uint8_t *smA = stage_out + kEpiWarps * kEpi * kOutBox;
    uint8_t *dig = smA + a.tc_a_stages * a.tc_a_max_bytes;
    uint8_t *raw = dig + a.tc_dig_stages * kDigStageBytes;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kMaxAStages; ++s) {
            mbar_init(&sh.a_full[s], 1);
            mbar_init(&sh.a_empty[s], 1);
        }
        mbar_init(&sh.drain, 1);
        for (uint32_t s = 0; s < kMaxRawStages; ++s) {
            mbar_init(&sh.raw_full[s], 1);
            mbar_init(&sh.raw_empty[s], kConvWarps);
        }
        for (uint32_t s = 0; s < kMaxDigStages; ++s) {
            mbar_init(&sh.dig_full[s], kConvWarps);
            mbar_init(&sh.dig_empty[s], 1);
        }
        for (uint32_t s = 0; s < kAccStages; ++s) {
            mbar_init(&sh.acc_full[s], 1);
            mbar_init(&sh.acc_empty[s], kEpiWarps);
        }
        sh.abort = 0;
        fence_mbar_init();
    }
    if (kRotated && threadIdx.x < kOutBox / 16) {
        sts_v4(smem_addr(smem + kZeroBox) + threadIdx.x * 16, 0, 0, 0, 0);
        fence_proxy_async_smem();
    }
    if (warp == kMmaWarp) tmem_alloc(&sh.tmem_base, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;

    if (warp == kDigitWarp) {
        // -------------------------------------------- coefficient digit loads
        if (lane == 0) {
            Ring ra;
            uint32_t loads = 0;
            for (Units w(a); w.valid(a); w.next(a)) {
                const PlanBlock *h = w.header(a);
                const uint32_t bytes = uint32_t(tc_a_bytes(h->n_groups));
                const uint8_t *src = a.tc_a + uint64_t(h->group_begin) * 16;
                if (ra.round > 0 && !tc_wait(&sh.abort, &sh.a_empty[ra.s], (ra.round - 1) & 1u, a.err)) break;
                mbar_arrive_expect_tx(&sh.a_full[ra.s], bytes);
                bulk_g2s(smA + ra.s * a.tc_a_max_bytes, src, bytes, &sh.a_full[ra.s]);
                ++loads;
                ra.next(a.tc_a_stages);
                if (kRotated && a.tc_store_map) {
                    // the unit's share of the slices that are zeros, where whole
                    // boxes go out (the epilogue stores the others)
                    const uint32_t z0 = w.z0(a), z1 = w.z1(a), lo = h->out_lo, hi = h->out_hi;
                    for (uint32_t o = lo; o + 32 <= hi && z0 < z1; o += 32) {
                        if (o < a.out_lo || uint64_t(o) + 32 > a.out_hi) continue;
                        for (uint32_t c = z0 * kN; c < z1 * kN; c += 32)
                            tma_store_2d(&maps.out, int32_t(c), int32_t(o - uint32_t(a.out_row_base)),
                                         smem_addr(smem + kZeroBox));
                    }
                    bulk_commit();
                }
            }
            if (kRotated) bulk_wait();
            // let every copy land: the last fill of each buffer (immediate when nothing aborted)
            for (uint32_t k = 1; k <= a.tc_a_stages && k <= loads; ++k) {
                const uint32_t j = loads - k;
                mbar_wait_bounded(&sh.a_full[j % a.tc_a_stages], (j / a.tc_a_stages) & 1u, nullptr);
            }
        }
        __syncwarp();
    } else if (warp >= kProducerWarp && warp < kMmaWarp) {
        // ------------------------------------------------------------ producer
        // The block header is read two units ahead and the rows one unit
        // ahead, so that the loop below issues copies and nothing else: with
        // the lookups in it, it took 850 cycles per chunk and bound the kernel.
        struct Rows {
            uint32_t n_slots, runs, n_chunks;  // runs: the block's consecutive-chunk mask
            uint32_t row[kMaxChunks], rot[kMaxChunks];  // lane i: slot i of each chunk
        };
        const bool leader = elect_one();
        // Each of the producers takes its chunks in turn (the raw stages are a
        // multiple of both counts).  Copying rows one by one is worth the
        // second (10 neighbours over permuted rows: one 0.327, two 0.261 ms);
        // boxes are not (headline 0.421 and 0.430 ms).
        const uint32_t me = warp - kProducerWarp;
        uint32_t *rows = kRotated ? rot.rows[me] : sh.rows[me], *rots = rot.rots[me];
        uint32_t turn = 0;
        Units head(a);
        PlanBlock blk{};
        Rows next{};
        auto fetch_header = [&]() {
            if (head.valid(a)) blk = *head.header(a);
            head.next(a);
        };
        auto fetch_rows = [&]() {  // of the block header last read
            next.n_slots = a.n_rows ? blk.n_slots : 0;
            next.runs = blk.term_begin;
            next.n_chunks = (blk.n_groups + kChunk - 1) / kChunk;
#pragma unroll
            for (uint32_t c = 0; c < kMaxChunks; ++c)
                if (kChunk * c + lane < blk.n_slots) {
                    const PlanSlot slot = a.slots[blk.slot_begin + kChunk * c + lane];
                    next.row[c] = slot.row;
                    if (kRotated) next.rot[c] = slot.rot;
                }
        };
        fetch_header();
        fetch_rows();
        fetch_header();
        Ring rr, last;
        bool any = false;
        // Lets the copies land: this warp's last ones (immediate when nothing
        // aborted; every earlier one was waited for by way of its stage's
        // converters or is behind one of these).
        auto land = [&]() {
            if (leader)
                for (uint32_t s = me; s < a.tc_raw_stages; s += kProducers) {
                    // the stage's last phase that this warp filled
                    const uint32_t filled = last.round + (s <= last.s ? 1u : 0u);
                    if (any && filled) mbar_wait_bounded(&sh.raw_full[s], (filled - 1) & 1u, nullptr);
                }
            cp_async_wait_all();
        };
        for (Units w(a); w.valid(a); w.next(a)) {
            const Rows x = next;
            fetch_rows();
            fetch_header();
            // rows as held at a.in; 0, reported, for one outside it (and 0 past the
            // block's slots: whatever lanes are left copy rows inside the input).
            // With tc_rows_partial a row outside is one that only outputs not
            // wanted read, and any other does.
            __syncwarp();
#pragma unroll
            for (uint32_t c = 0; c < kMaxChunks; ++c) {
                uint32_t r = x.row[c] - a.row_base;
                if (r >= a.n_rows) {
                    if (kChunk * c + lane < x.n_slots && !(kRotated && a.tc_rows_partial))
                        report_error(a.err, kDevBadIndex);
                    r = 0;
                }
                rows[kChunk * c + lane] = r;
                if (kRotated) rots[kChunk * c + lane] = x.rot[c];
            }
            __syncwarp();
            // lane c: the first row of chunk c; the chunks that one tensor copy
            // loads (consecutive rows, all inside the input)
            const uint32_t first = rows[kChunk * min(lane, kMaxChunks - 1)];
            const uint32_t n_here = kChunk * lane < x.n_slots ? min(kChunk, x.n_slots - kChunk * lane) : 0u;
            const uint32_t boxes = __ballot_sync(0xFFFFFFFFu, n_here && a.tc_use_map && ((x.runs >> lane) & 1u) &&
                                                                  first < a.n_rows && n_here <= a.n_rows - first);
            const uint32_t s1 = w.s1(a);
            for (uint32_t sl = w.s0(a); sl < s1; ++sl) {
                const uint32_t c0 = sl * kN;
#pragma unroll 1
                for (uint32_t c = 0; c < x.n_chunks; ++c) {
                    const bool mine = turn == me;
                    if (++turn == kProducers) turn = 0;
                    if (!mine) {
                        rr.next(a.tc_raw_stages);
                        continue;
                    }
                    // undefined where lane c has given up: only a coordinate, which the map bounds
                    const int32_t r0 = int32_t(__shfl_sync(0xFFFFFFFFu, first, c));
                    uint64_t *full = &sh.raw_full[rr.s];
                    uint8_t *dst = raw + rr.s * kRawStageBytes;
                    if (rr.round > 0 && !tc_wait(&sh.abort, &sh.raw_empty[rr.s], (rr.round - 1) & 1u, a.err)) {
                        land();
                        return;  // the others of the warp do without this lane
                    }
                    if ((boxes >> c) & 1u) {
                        if (leader) {
                            if (kRotated) rot.any[rr.s] = 0;
                            fence_proxy_async_smem();  // after the converters' reads of the stage
                            mbar_arrive_expect_tx(full, kRawStageBytes);
                            tma_load_2d(dst, &maps.rows, int32_t(c0), r0, full);
                        }
                    } else if (kRotated && x.n_slots > kChunk * c) {
                        const uint32_t n = min(kChunk, x.n_slots - kChunk * c);
                        const uint32_t *r = rows + kChunk * c, *m = rots + kChunk * c;
                        if (a.tc_rot_bytes == 16) load_rotated<16>(a, r, m, n, c0, smem_addr(dst), lane);
                        else if (a.tc_rot_bytes == 8) load_rotated<8>(a, r, m, n, c0, smem_addr(dst), lane);
                        else load_rotated<4>(a, r, m, n, c0, smem_addr(dst), lane);
                        // columns that stay in the polynomial, from c0 on
                        const uint32_t to_end = a.N - (c0 & (a.N - 1));
                        const uint32_t stay = lane < n ? to_end - min(m[lane], to_end) : kN;
                        rot.from[rr.s][lane] = stay;
                        const bool any = __any_sync(0xFFFFFFFFu, stay < kN);
                        if (lane == 0) rot.any[rr.s] = any;
                        cp_async_arrive(full);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(full);
                    } else if (x.n_slots > kChunk * c) {
                        load_rows(a, rows + kChunk * c, min(kChunk, x.n_slots - kChunk * c), c0, smem_addr(dst), full, lane);
                    } else if (leader) {
                        if (kRotated) rot.any[rr.s] = 0;
                        mbar_arrive(full);  // rows of padding only: their coefficients are zero
                    }
                    __syncwarp();
                    last = rr;
                    any = true;
                    rr.next(a.tc_raw_stages);
                }
            }
        }
        land();
        __syncwarp();
    } else if (warp >= kConvWarp0) {
        // ---------------------------------------------------------- converters
        // unit q of a chunk: rows 8 (q / 64) .. + 7 of column q % 64.  A warp's
        // loads are 32 consecutive words, its stores 32 consecutive 16-byte rows.
        constexpr uint32_t kTeamThreads = 32 * kConvWarps, kUnits = kN * (kChunk / 8) / kTeamThreads;
        const uint32_t team = (warp - kConvWarp0) / kConvWarps;
        const uint32_t tid = (warp - kConvWarp0) % kConvWarps * 32 + lane;
        uint32_t turn = 0;
        Ring rr, rd;
        bool ok = true;
        UnitDepths depths(a);
        for (Units w(a); ok && w.valid(a); w.next(a)) {
            const uint32_t k_pad = depths.next(a);
            for (uint32_t n = w.s1(a) - w.s0(a); ok && n > 0; --n) {
                for (uint32_t k0 = 0; k0 < k_pad; k0 += kChunk) {
                    const bool mine = turn == team;
                    if (++turn == kConv) turn = 0;
                    if (!mine) {
                        rr.next(a.tc_raw_stages);
                        rd.next(a.tc_dig_stages);
                        continue;
                    }
                    if (!(ok = tc_warp_wait(&sh.abort, &sh.raw_full[rr.s], rr.round & 1u, a.err, lane))) break;
                    const uint32_t groups = min(kChunk, k_pad - k0) / 8;
                    const uint32_t src = smem_addr(raw + rr.s * kRawStageBytes);
                    const uint32_t dst = smem_addr(dig + rd.s * kDigStageBytes);
                    // All of the raw stage's words first: it is free once they
                    // are here.  Volatile loads: with plain ones the compiler
                    // moved them below the arrival and the wait that follow.
                    uint32_t w[kUnits][8];
                    const bool negate = kRotated && *reinterpret_cast<volatile uint32_t *>(&rot.any[rr.s]) != 0;
#pragma unroll
                    for (uint32_t x = 0; x < kUnits; ++x) {
                        const uint32_t q = x * kTeamThreads + tid, g = q / kN, col = q % kN;
                        if (g >= groups) break;
#pragma unroll
                        for (uint32_t r = 0; r < 8; ++r)
                            asm volatile("ld.volatile.shared.u32 %0, [%1];"
                                         : "=r"(w[x][r])
                                         : "r"(src + ((8 * g + r) * kN + col) * 4)
                                         : "memory");
                        if (negate) {
                            const uint32_t at = smem_addr(&rot.from[rr.s][8 * g]);
                            const uint4 f0 = lds_v4_ordered(at), f1 = lds_v4_ordered(at + 16);
                            const uint32_t from[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
                            for (uint32_t r = 0; r < 8; ++r)
                                if (col >= from[r]) w[x][r] = 0u - w[x][r];
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.raw_empty[rr.s]);
                    if (rd.round > 0 &&
                        !(ok = tc_warp_wait(&sh.abort, &sh.dig_empty[rd.s], (rd.round - 1) & 1u, a.err, lane)))
                        break;
#pragma unroll
                    for (uint32_t x = 0; x < kUnits; ++x) {
                        const uint32_t q = x * kTeamThreads + tid, g = q / kN, col = q % kN;
                        if (g >= groups) break;
                        uint32_t p[4][4];
#pragma unroll
                        for (uint32_t r = 0; r < 4; ++r) {
                            const uint32_t lo = __byte_perm(w[x][2 * r], w[x][2 * r + 1], 0x5140);
                            const uint32_t hi = __byte_perm(w[x][2 * r], w[x][2 * r + 1], 0x7362);
                            p[0][r] = __byte_perm(lo, 0u, 0x4140);
                            p[1][r] = __byte_perm(lo, 0u, 0x4342);
                            p[2][r] = __byte_perm(hi, 0u, 0x4140);
                            p[3][r] = __byte_perm(hi, 0u, 0x4342);
                        }
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i)
                            sts_v4(dst + g * kGroupBytes + (i * kN + col) * 16, p[i][0], p[i][1], p[i][2], p[i][3]);
                    }
                    fence_proxy_async_smem();  // the digits are read by the tensor cores (async proxy)
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.dig_full[rd.s]);
                    rr.next(a.tc_raw_stages);
                    rd.next(a.tc_dig_stages);
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ----------------------------------------------------------------- MMA
        // Each lane leaves by its own verdict: nothing in the loop waits for the
        // other lanes.
        Ring rd, ra, rt;
        bool ok = true;
        const bool leader = elect_one();
        const uint64_t a_desc = umma_desc(smem_addr(smA), 2048, 128);
        const uint64_t d_desc = umma_desc(smem_addr(dig), kGroupBytes, 128);
        UnitDepths depths(a);
        for (Units w(a); ok && w.valid(a); w.next(a)) {
            const uint32_t k_pad = depths.next(a);
            if (!(ok = tc_wait(&sh.abort, &sh.a_full[ra.s], ra.round & 1u, a.err))) break;
            const uint64_t a_unit = a_desc + ra.s * (a.tc_a_max_bytes / 16);
            const uint32_t plane = k_pad * 16;  // 16-byte units per coefficient digit plane
            for (uint32_t n = w.s1(a) - w.s0(a); ok && n > 0; --n) {
                if (rt.round > 0 && !(ok = tc_wait(&sh.abort, &sh.acc_empty[rt.s], (rt.round - 1) & 1u, a.err))) break;
                tc_fence_after();
                const uint32_t d0 = tmem + rt.s * (4 * kN);
                uint64_t a0 = a_unit;
                for (uint32_t k0 = 0; k0 < k_pad; k0 += kChunk) {
                    if (!(ok = tc_wait(&sh.abort, &sh.dig_full[rd.s], rd.round & 1u, a.err))) break;
                    tc_fence_after();
                    const uint64_t b0 = d_desc + rd.s * (kDigStageBytes / 16);
                    if (leader) {
                        umma_f16(d0, a0, b0, kIdescAll, k0 > 0 ? 1u : 0u);
                        umma_f16(d0 + kN, a0 + plane, b0, kIdescHigh, 1u);
                        if (k_pad - k0 > 16) {
                            umma_f16(d0, a0 + 256, b0 + 2 * kGroupBytes / 16, kIdescAll, 1u);
                            umma_f16(d0 + kN, a0 + plane + 256, b0 + 2 * kGroupBytes / 16, kIdescHigh, 1u);
                        }
                        umma_commit(&sh.dig_empty[rd.s]);
                        if (k0 + kChunk >= k_pad) {
                            umma_commit(&sh.acc_full[rt.s]);
                            if (n == 1) umma_commit(&sh.a_empty[ra.s]);
                        }
                    }
                    a0 += 512;
                    rd.next(a.tc_dig_stages);
                }
                rt.next(kAccStages);
            }
            ra.next(a.tc_a_stages);
        }
        // every MMA issued has completed before TMEM is released
        if (leader) umma_commit(&sh.drain);
        mbar_wait_bounded(&sh.drain, 0, nullptr);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        const uint32_t team = warp / kEpiWarps, quadrant = warp % 4;  // tiles taken, TMEM lanes
        const uint32_t half = (warp / 4) % 2;                         // columns [32 half, + 32) of the tile
        const uint32_t row = quadrant * 32 + lane;
        const uint32_t stage = smem_addr(stage_out + warp * kOutBox);
        Ring rt;  // accumulator stage of the tile
        uint32_t turn = 0, lwe_next = 0xFFFFFFFFu;
        bool ok = true;
        // the unit's outputs are read two units ahead, this lane's constants one
        Units head(a);
        uint32_t lo = 0, hi = 0, next_o = 0;
        bool next_has = false;
        TcOut next_oc{};
        auto fetch_header = [&]() {
            lo = hi = 0;
            if (head.valid(a)) {
                lo = head.header(a)->out_lo;
                hi = head.header(a)->out_hi;
            }
            head.next(a);
        };
        auto fetch_constants = [&]() {  // of the block header last read
            next_o = lo + row;
            next_has = next_o < hi && next_o >= a.out_lo && next_o < a.out_hi;
            next_oc = TcOut{0, 0, 0.75f, 0.75f};
            if (next_has) next_oc = a.tc_out[next_o];
        };
        fetch_header();
        fetch_constants();
        fetch_header();
        for (Units w(a); ok && w.valid(a); w.next(a)) {
            const uint32_t o = next_o;
            const bool has = next_has;
            const TcOut oc = next_oc;
            fetch_constants();
            fetch_header();
            const uint32_t add0 = oc.offset - kMagicSum;
            uint8_t *orow = has ? a.out + (a.out_row_map ? uint64_t(a.out_row_map[o]) : uint64_t(o) - a.out_row_base) *
                                              a.out_stride
                                : nullptr;
            // the warp's 32 outputs are all wanted: whole boxes go out
            const bool boxes = a.tc_store_map && __all_sync(0xFFFFFFFFu, has);
            const uint32_t s1 = w.s1(a);
            for (uint32_t sl = w.s0(a); ok && sl < s1; ++sl) {
                const Ring at = rt;
                rt.next(kAccStages);
                const bool mine = turn == team;
                if (++turn == kEpi) turn = 0;
                if (!mine) continue;
                if (!(ok = tc_team_wait<32 * kEpiWarps>(1 + team, warp % kEpiWarps == 0 && lane == 0, &sh.abort,
                                                        &sh.acc_full[at.s], at.round & 1u, a.err)))
                    break;
                tc_fence_after();
                const uint32_t base = tmem + ((quadrant * 32) << 16) + at.s * (4 * kN) + 32 * half;
                // this warp's 32 columns, from c0; `valid` of them inside the row
                const uint32_t c0 = sl * kN + 32 * half;
                const uint32_t valid = c0 < a.row_words ? min(32u, a.row_words - c0) : 0u;
                // columns that take the bias, and that are zeroed
                uint32_t bias_cols = 0, zero_cols = 0;
                if (a.form == kFormTrlwe) {
                    bias_cols = columns_in(c0, a.N, a.N + a.num_samples);
                    zero_cols = columns_in(c0, a.N + a.region_size, 2 * a.N);
                } else {
                    // body words: columns c with c % n1 == n; lwe_next is the first from c0 on
                    if (lwe_next < c0 || lwe_next - c0 >= a.lwe_n1) lwe_next = c0 + (a.lwe_n1 - 1u) - c0 % a.lwe_n1;
                    for (uint32_t c = lwe_next - c0; c < 32; c += a.lwe_n1) bias_cols |= 1u << c;
                }
                const bool mixed = zero_cols != 0 || (bias_cols != 0 && bias_cols != 0xFFFFFFFFu);
                const uint32_t add_all = (bias_cols == 0xFFFFFFFFu ? oc.bias : 0u) + add0;
#pragma unroll
                for (uint32_t cc = 0; cc < 4; ++cc) {
                    uint32_t d[4][8], v[8];
#pragma unroll
                    for (uint32_t s = 0; s < 4; ++s) tmem_ld8(base + s * kN + cc * 8, d[s]);
                    if (cc == 0) {
                        if (lane == 0) bulk_wait_read<0>();  // the box stored last has been read
                        __syncwarp();
                    }
                    tmem_wait_ld();
                    if (cc == 3) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.acc_empty[at.s]);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < 8; j += 2) {
                        add2(d[0][j], d[0][j + 1], oc.m0);
                        add2(d[1][j], d[1][j + 1], oc.m1);
                        add2(d[2][j], d[2][j + 1], oc.m1);
                        add2(d[3][j], d[3][j + 1], oc.m1);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        v[j] = (((d[3][j] << 24) + add_all) + (d[2][j] << 16)) + ((d[1][j] << 8) + d[0][j]);
                    if (mixed) {
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j) {
                            const uint32_t bit = 1u << (cc * 8 + j);
                            if (bias_cols != 0xFFFFFFFFu && (bias_cols & bit)) v[j] += oc.bias;
                            if (zero_cols & bit) v[j] = 0u;
                        }
                    }
                    // 16-byte piece p of the box's row goes to piece p ^ (row % 8)
#pragma unroll
                    for (uint32_t j = 0; j < 8; j += 4)
                        sts_v4(stage + lane * 128 + ((cc * 2 + j / 4) ^ (lane % 8)) * 16, v[j], v[j + 1], v[j + 2],
                               v[j + 3]);
                }
                if (boxes) {
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && valid) {
                        tma_store_2d(&maps.out, int32_t(c0), int32_t(o - uint32_t(a.out_row_base)), stage);
                        bulk_commit();
                    }
                    continue;
                }
                __syncwarp();
                // row by row: eight lanes store 128 bytes of one row, four
                // rows at a time; row r's address comes from lane r
                const uint32_t p = lane % 8;
                const uint64_t mine_row = reinterpret_cast<uint64_t>(orow);
#pragma unroll 1
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint32_t r = 4 * i + lane / 8;
                    const uint64_t dst = __shfl_sync(0xFFFFFFFFu, mine_row, r);
                    const uint4 w = lds_v4_ordered(stage + r * 128 + (p ^ (r % 8)) * 16);
                    if (!dst || 4 * p >= valid) continue;
                    uint32_t *g = reinterpret_cast<uint32_t *>(dst) + c0 + 4 * p;
                    if (4 * p + 4 <= valid) {
                        stg_cs_v4(g, make_int4(int(w.x), int(w.y), int(w.z), int(w.w)));
                    } else {
                        g[0] = w.x;
                        if (4 * p + 1 < valid) g[1] = w.y;
                        if (4 * p + 2 < valid) g[2] = w.z;
                    }
                }
                __syncwarp();  // the warp has read its staged rows before they are overwritten
            }
            if (!kRotated) continue;
            // the unit's share of the slices that are zeros; the teams in turn
            const uint32_t z0 = w.z0(a), z1 = w.z1(a);
            if (!ok || boxes || z0 + team >= z1) continue;
            for (uint32_t i = 0; i < 8; ++i) {
                const uint64_t dst = __shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(orow), 4 * i + lane / 8);
                if (!dst) continue;
                for (uint32_t sl = z0 + team; sl < z1; sl += kEpi) {
                    const uint32_t c = sl * kN + 32 * half + 4 * (lane % 8);
                    for (uint32_t e = c; e < min(c + 4, a.row_words); ++e) reinterpret_cast<uint32_t *>(dst)[e] = 0u;
                }
            }
        }
        if (lane == 0) bulk_wait();  // the stored boxes are written
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemCols);
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// A 2D tensor of uint32 (`words` columns x `rows` rows, `stride` bytes between
// rows) read or written in boxes.  False when it cannot be encoded (the
// kernel then copies row by row).
bool encode_rows_map(const uint8_t *base, uint64_t words, uint64_t rows, uint64_t stride, uint32_t box_words,
                     uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMap *map) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || rows == 0 || rows > 0x7FFFFFFFull || stride % 16 || (reinterpret_cast<uintptr_t>(base) & 15u))
        return false;
    const cuuint64_t dims[2] = {words, rows};
    const cuuint64_t strides[1] = {stride};
    const cuuint32_t box[2] = {box_words, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t *>(base), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

size_t tc_smem_bytes(uint32_t max_k_pad, bool rotated) {
    const TcShape *x = tc_shape(max_k_pad, rotated);
    return x ? x->smem(max_k_pad, rotated) : SIZE_MAX;
}

bool tc_digits_ahead(uint32_t max_k_pad, bool rotated) {
    const TcShape *x = tc_shape(max_k_pad, rotated);
    return x && x->a_stages > 1;
}

cudaError_t configure_tc_kernel(size_t max_smem) {
    for (auto *fn : {k_score_tc<2, 2, 2, 1>, k_score_tc<2, 2, 2, 2>, k_score_tc<1, 3, 4, 1>, k_score_tc<1, 3, 4, 2>,
                     k_score_tc<1, 2, 4, kTcRotProducers, true>}) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(max_smem));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_score_tc(const ScoreArgs &a_in, uint32_t ctas, cudaStream_t stream) {
    if (a_in.n_units == 0) return cudaSuccess;
    if (a_in.accumulate || a_in.digest || a_in.units_per_block == 0 || a_in.unit_slices == 0)
        return cudaErrorInvalidValue;
    ScoreArgs a = a_in;
    const uint32_t k = a.tc_a_max_bytes / uint32_t(tc_a_bytes(1));
    const bool rotated = a.tc_rot_bytes != 0;
    const TcShape *shape = tc_shape(k, rotated);
    if (!shape) return cudaErrorInvalidValue;
    a.tc_a_stages = shape->a_stages;
    a.tc_dig_stages = shape->dig_stages;
    a.tc_raw_stages = shape->raw_stages;
    if (a.tc_producers == 0 || (rotated ? a.tc_producers != kTcRotProducers : a.tc_producers > kTcMaxProducers))
        return cudaErrorInvalidValue;
    TcMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    // (no boxes over rows that are not all there)
    a.tc_use_map = !a.tc_rows_partial && encode_rows_map(a.in, a.row_words, a.n_rows, a.in_stride, kN, kChunk,
                                                         CU_TENSOR_MAP_SWIZZLE_NONE, &maps.rows);
    a.tc_store_map = !a.out_row_map && a.out_lo >= a.out_row_base &&
                     encode_rows_map(a.out, a.row_words, a.out_hi - a.out_row_base, a.out_stride, 32, 32,
                                     CU_TENSOR_MAP_SWIZZLE_128B, &maps.out);
    const uint32_t grid = ctas < a.n_units ? ctas : a.n_units;
    a.unit_step_blocks = grid / a.units_per_block;
    a.unit_step_parts = grid % a.units_per_block;
    const bool two = a.tc_producers == 2;
    auto *fn = rotated           ? k_score_tc<1, 2, 4, kTcRotProducers, true>
               : shape->epi == 2 ? (two ? k_score_tc<2, 2, 2, 2> : k_score_tc<2, 2, 2, 1>)
                               : (two ? k_score_tc<1, 3, 4, 2> : k_score_tc<1, 3, 4, 1>);
    const uint32_t threads = tc_threads(shape->epi, shape->conv, shape->conv_warps, a.tc_producers);
    fn<<<grid, threads, shape->smem(k, rotated), stream>>>(a, maps);
    return cudaGetLastError();
}

}  // namespace idash
