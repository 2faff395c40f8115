// Bounded waits of the roles that share a CTA (score_tc.cu, key_product.cu,
// intpoly.cu): by one thread, by a warp and by a team of warps.
#pragma once

#include "common.cuh"

namespace idash {

// Bounded wait that also ends when another role raised the CTA's abort flag.
// For one thread: around an expiry the lanes of a warp can take the phase, the
// flag and the clock in different orders and come to different verdicts.  Where
// a warp runs its loop whole, a lane without what it waited for therefore
//   - leaves the loop, if nothing in it waits for the other lanes; or
//   - exits (return), since a warp's barriers, shuffles and votes and the CTA's
//     barriers are for the threads that have not exited (values from lanes that
//     have are undefined: no address depends on them but by a tensor map, which
//     bounds it).
// (One verdict for all by a shuffle or vote after each wait: 0.2 to 2.6% of a
// scoring pass with TRLWE rows, 1.5 to 5% with LWE rows.)
__device__ __forceinline__ bool tc_wait(uint32_t *abort, uint64_t *bar, uint32_t parity, uint32_t *err,
                                        long long limit = kWaitLimitCycles) {
    if (mbar_try_wait(bar, parity)) return true;
    volatile uint32_t *flag = abort;
    const long long t0 = clock64();
    for (;;) {
        // a few tries between looks at the flag and the clock: waiting warps
        // share the issue slots with working ones
#pragma unroll 1
        for (int i = 0; i < 8; ++i)
            if (mbar_try_wait_sleep(bar, parity, 20000u)) return true;
        if (*flag != 0) return false;
        if (clock64() - t0 > limit) {
            report_error(err, kDevTimeout);
            *flag = 1u;
            return false;
        }
    }
}

// Lane 0 waits, the warp follows its verdict.
__device__ __forceinline__ bool tc_warp_wait(uint32_t *abort, uint64_t *bar, uint32_t parity, uint32_t *err,
                                             uint32_t lane) {
    uint32_t ok = 1;
    if (lane == 0) ok = tc_wait(abort, bar, parity, err) ? 1u : 0u;
    return __shfl_sync(0xFFFFFFFFu, ok, 0) != 0;
}

// Whether `ok` holds for all kThreads threads of a team of warps, at named
// barrier `id` (1 .. 15).  A team waits with one thread polling and the others
// standing here, where they take no issue slots.  (Every warp polling for
// itself made up half of the instructions that the scoring kernel issued.)
template <int kThreads>
__device__ __forceinline__ bool tc_team_and(uint32_t id, bool ok) {
    uint32_t r = ok ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %0, 0;\n\t"
        "barrier.cta.red.and.pred q, %1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "+r"(r)
        : "r"(id), "n"(kThreads)
        : "memory");
    return r != 0;
}

template <int kThreads>
__device__ __forceinline__ bool tc_team_wait(uint32_t id, bool polls, uint32_t *abort, uint64_t *bar, uint32_t parity,
                                             uint32_t *err, long long limit = kWaitLimitCycles) {
    return tc_team_and<kThreads>(id, !polls || tc_wait(abort, bar, parity, err, limit));
}

}  // namespace idash
