// time_step.cuh -- the end of the constitutive kernel: the critical timestep
// minimum (MCM/mcm_calccritts.f90:82-85), the dt update
// (MCM/mcm_solution.f90:58-62) and termination test (:101) on the device.
#pragma once
#include "kernels.h"

namespace mcm {

// The order of doubles as that of unsigned integers, and back.
__host__ __device__ inline unsigned long long order_bits(unsigned long long b) {
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__host__ __device__ inline unsigned long long unorder_bits(unsigned long long b) {
    return (b >> 63) ? b & 0x7fffffffffffffffull : ~b;
}

// Called by thread 0 of every block with the block's minimum.  The minimum over
// the blocks is an integer atomic, whose result does not depend on their order;
// the block that ends last advances the time scalars.  (A launch of its own
// before: 7 to 9 us a step.)
__device__ __forceinline__ void finish_critts(const StepArgs &a, double block_min) {
    atomicMin(a.crit_bits, order_bits((unsigned long long)__double_as_longlong(block_min)));
    __threadfence();
    if (atomicAdd(a.crit_ticket, 1) != (int)gridDim.x - 1) return;
    __threadfence();
    DevTime *t = a.time;
    if (*(volatile int *)&a.status->code) return;
    const double m = __longlong_as_double((long long)unorder_bits(*(volatile unsigned long long *)a.crit_bits));
    t->critts = m;
    if (a.prm.h_opt) {
        // the largest h of this step's mcm_update_h becomes the next grid's hmax
        // (kept when no particle was at or above its cut-off pressure)
        volatile unsigned long long *bid = reinterpret_cast<volatile unsigned long long *>(a.hmax + 1);
        const unsigned long long b = *bid;
        if (b) a.hmax[0] = __longlong_as_double(static_cast<long long>(b));
        *bid = 0ull;
    }
    if (!a.split_mode) {
        t->dtold = t->dt;
        double dt = a.prm.tssf * m;
        double lim = 1.1 * t->dtold;
        t->dt = (lim < dt) ? lim : dt;
        t->ptime = t->ptime + t->dt;
        if (t->ptime - t->dt >= t->endtime) t->ended = 1;
    }
}

}  // namespace mcm
