// swe_clock.cuh -- the bookkeeping between two steps of forward(): shared by
// the clock kernel (swe_driver.cu) and the stage-2 kernels of a clocked step,
// which advance the clock while the stage runs.  The arithmetic is the
// reference's whatever the including file's contraction: double-precision
// elapsed / remaining time, float32 max_dt, float32 interpolation of the
// boundary series.
#pragma once

#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "swe_common.cuh"

namespace swe {
namespace {

// SWE2D._interpolate_dynamic_boundary (src/solver.py:391-415) in float32:
// index = searchsorted(times, t, right=False) clamped to [1, n-1].
__device__ inline float interpolate_level(const float* times, const float* levels, int n, float t) {
    if (n == 1) return levels[0];
    int lo = 0, hi = n;
    while (lo < hi) {  // first index with times[i] >= t
        const int mid = (lo + hi) >> 1;
        if (times[mid] < t) lo = mid + 1;
        else hi = mid;
    }
    const int idx = min(max(lo, 1), n - 1);
    const float t0 = times[idx - 1], t1 = times[idx];
    const float w0 = levels[idx - 1], w1 = levels[idx];
    const float weight = __fdiv_rn(__fsub_rn(t, t0), fmaxf(__fsub_rn(t1, t0), FLT_EPSILON));
    return __fadd_rn(w0, __fmul_rn(weight, __fsub_rn(w1, w0)));
}

// Takes the clock past the step that ran with time step dt and status bits st
// (solver.py:627-632, :765-768), if it was active; whether it completed.
__device__ __forceinline__ bool clock_finish_step(swe_clock& cl, uint32_t st, float dt) {
    if (!cl.active) return false;
    cl.last_dt = dt;
    if (st & (SWE_S_NONFINITE_STATE | SWE_S_NONFINITE_DT | SWE_S_NONPOSITIVE_DT)) {
        cl.state = SWE_CLOCK_FAILED;
        cl.dt_status = st;
        cl.active = 0;
        return false;
    }
    double elapsed = cl.elapsed + (double)dt;
    if (elapsed > cl.duration && elapsed - cl.duration <= cl.tolerance) elapsed = cl.duration;
    cl.elapsed = elapsed;
    cl.steps += 1;
    return true;
}

// Sets up the next step (solver.py:741-760), if there is one.
__device__ __forceinline__ void clock_set_up(swe_clock& cl, const float* series_t, const float* series_w, int nseries,
                                             float* level_out, uint32_t* red) {
    if (cl.state != SWE_CLOCK_RUNNING) {
        cl.active = 0;
        return;
    }
    // The loop runs out of iterations before it checks the remaining time
    // again, so max_steps is tested first.
    const double remaining = cl.duration - cl.elapsed;
    if (cl.steps >= cl.max_steps) {
        cl.state = SWE_CLOCK_MAXSTEPS;
        cl.active = 0;
    } else if (remaining <= cl.tolerance) {
        cl.state = SWE_CLOCK_DONE;
        cl.active = 0;
    } else {
        double step_max_dt = remaining;
        if (cl.max_dt_cap > 0.0 && cl.max_dt_cap < remaining) step_max_dt = cl.max_dt_cap;
        cl.max_dt = (float)step_max_dt;
        if (nseries > 0) {
            const float lev = interpolate_level(series_t, series_w, nseries, (float)(cl.start + cl.elapsed));
            cl.level = lev;
            level_out[0] = lev;
        }
        red[0] = 0u;
        red[1] = 0u;
        red[2] = 0u;
        cl.active = 1;
    }
}

}  // namespace
}  // namespace swe
