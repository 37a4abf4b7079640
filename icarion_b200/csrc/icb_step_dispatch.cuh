// icb_step_dispatch.cuh — maps runtime (integrator, collision, field, B)
// choices onto the compiled template instances of k_step.
#pragma once
#include <cuda_runtime.h>
#include "icb_step_kernel.cuh"

namespace icb {

// Whether the float RF / time-dependent kernel should run with room for 24
// resident warps per SM (80 registers, more of them spilled) instead of 20
// (96): when the launch then takes fewer rounds of resident warps.  Every warp
// runs the same number of steps, so a round that is nearly empty still costs
// most of a round.  Time with 24 over time with 20, trap of 22 to 72 warps of
// ions per SM, 300 steps:
//   2 rounds -> 1: 0.62 to 0.98 in every form (mixed and hi/lo, Boris and
//     RK4, with and without B, collisions and a time-dependent field);
//   3 -> 2 and 4 -> 3 (`later`): mixed Boris with collisions 0.83 to 0.98,
//     without collisions or B 0.91 to 1.02, mixed RK4 with collisions in a
//     constant-voltage field 0.88 to 0.99.  The others spill more than the
//     round saves: RK4 without collisions 1.08 to 1.24, RK4 in a
//     time-dependent field 0.98 to 1.08, no collisions with B 1.03 to 1.11,
//     hi/lo 0.88 (network) to 1.16 (no collisions);
//   the same number of rounds: 1.01 to 1.38.
inline bool more_warps(dim3 grid, dim3 block, bool later) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        return false;
    const uint64_t warps = static_cast<uint64_t>(grid.x) * (block.x / 32u);
    const uint64_t a = 20ull * static_cast<uint64_t>(sms), b = 24ull * static_cast<uint64_t>(sms);
    const uint64_t ra = (warps + a - 1) / a, rb = (warps + b - 1) / b;
    return rb < ra && (ra == 2u || (later && ra <= 4u));
}

template <int PREC, int INTEG, int COLL, int FIELD, bool MAG>
cudaError_t launch_one(const StepParams& p, dim3 grid, dim3 block, cudaStream_t s) {
    if constexpr (PREC != kPrecFP64 && FIELD == kFieldLinearRF) {
        constexpr bool kColl = COLL != kCollNone;
        bool tf = false;
        for (uint32_t e = 0; e < p.n_ens; ++e) tf = tf || p.ens[e].tf;
        const bool later = PREC == kPrecMixed && (INTEG == kBoris ? kColl || !MAG : kColl && !tf);
        if (p.do_push && p.do_collide && p.do_finalize && more_warps(grid, block, later)) {
            k_step<PREC, INTEG, COLL, FIELD, MAG, true, 6><<<grid, block, 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    if (p.do_push && p.do_collide && p.do_finalize)
        k_step<PREC, INTEG, COLL, FIELD, MAG, true><<<grid, block, 0, s>>>(p);
    else
        k_step<PREC, INTEG, COLL, FIELD, MAG, false><<<grid, block, 0, s>>>(p);
    return cudaGetLastError();
}

template <int PREC, int INTEG, int COLL>
cudaError_t dispatch_field(int field, bool mag, const StepParams& p, dim3 g, dim3 b, cudaStream_t s) {
    switch (field) {
        case kFieldUniform:
            return mag ? launch_one<PREC, INTEG, COLL, kFieldUniform, true>(p, g, b, s)
                       : launch_one<PREC, INTEG, COLL, kFieldUniform, false>(p, g, b, s);
        case kFieldLinear:
            return mag ? launch_one<PREC, INTEG, COLL, kFieldLinear, true>(p, g, b, s)
                       : launch_one<PREC, INTEG, COLL, kFieldLinear, false>(p, g, b, s);
        case kFieldLinearRF:
            return mag ? launch_one<PREC, INTEG, COLL, kFieldLinearRF, true>(p, g, b, s)
                       : launch_one<PREC, INTEG, COLL, kFieldLinearRF, false>(p, g, b, s);
        default:
            return cudaErrorNotSupported;
    }
}

template <int PREC, bool WITH_RK4>
cudaError_t dispatch_step(int integ, int coll, int field, bool mag, const StepParams& p,
                          dim3 g, dim3 b, cudaStream_t s) {
    if (integ == kBoris) {
        if (coll == kCollNone) return dispatch_field<PREC, kBoris, kCollNone>(field, mag, p, g, b, s);
        if (coll == kCollHSS) return dispatch_field<PREC, kBoris, kCollHSS>(field, mag, p, g, b, s);
        if (coll == kCollLangevin) return dispatch_field<PREC, kBoris, kCollLangevin>(field, mag, p, g, b, s);
        if (coll == kCollIPMTable) return dispatch_field<PREC, kBoris, kCollIPMTable>(field, mag, p, g, b, s);
        if (coll == kCollIPMMLP) return dispatch_field<PREC, kBoris, kCollIPMMLP>(field, mag, p, g, b, s);
        if (coll == kCollIPMQuad) {
            // the per-collision quadrature: built for the uniform drift field
            if (field != kFieldUniform || mag) return cudaErrorNotSupported;
            return launch_one<PREC, kBoris, kCollIPMQuad, kFieldUniform, false>(p, g, b, s);
        }
        if (coll == kCollHSSMix) return dispatch_field<PREC, kBoris, kCollHSSMix>(field, mag, p, g, b, s);
        if (coll == kCollEHSS) return dispatch_field<PREC, kBoris, kCollEHSS>(field, mag, p, g, b, s);
        if constexpr (PREC == kPrecFP64) {
            if (coll == kCollHSSPlain) return dispatch_field<PREC, kBoris, kCollHSSPlain>(field, mag, p, g, b, s);
        }
        return cudaErrorNotSupported;
    }
    if constexpr (WITH_RK4) {
        if (integ == kRK4) {
            if (coll == kCollNone) return dispatch_field<PREC, kRK4, kCollNone>(field, mag, p, g, b, s);
            if (coll == kCollHSS) return dispatch_field<PREC, kRK4, kCollHSS>(field, mag, p, g, b, s);
        }
    }
    return cudaErrorNotSupported;
}

}  // namespace icb
