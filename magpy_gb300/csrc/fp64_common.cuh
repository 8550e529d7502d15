// fp64_common.cuh -- helpers shared by the FP64-faithful kernels (sllg_fp64.cu,
// sllg_fp64_lanes.cu; both compiled with -fmad=false).
#pragma once
#include "mul_int.cuh"
#include "common.cuh"
#include "llg64.cuh"

namespace magpy {

// 0.0 + x without an FP64 instruction: x, but +0 for -0.
__device__ inline double plus_zero(double x)
{
    const bool mz = __double2hiint(x) == (int)0x80000000 && __double2loint(x) == 0;
    return mz ? 0.0 : x;
}

// The applied field at a step's two evaluation times, t = step dt and t + dt
// (Heun) or t + dt/2 (implicit midpoint).  An FP64 sine takes ~1300 cycles of
// a warp, as much as 20 other FP64 instructions, and every lane of a warp
// needs the same one when its members share their waveform and schedule: the
// lanes then compute consecutive steps, one each, and hand them out by
// shuffle.  (Same function, same argument, same bits.)  Members that do not
// share compute their own.
struct AppliedField {
    double a, b;      // this lane's step of the block
    int64_t base;     // steps before the block
    unsigned mask;    // lanes that share, 0: none
    int lanes;        // their number (they are lanes 0 .. lanes-1)

    __device__ inline void init(const MemberDev &d, bool share)
    {
        mask = 0;
        lanes = 0;
        base = 0;
        a = b = d.happ;  // constant field
        if (d.shape == FIELD_CONSTANT || !share) return;
        const unsigned act = __activemask();
        if ((act & (act + 1)) == 0 && act != 1u) {
            mask = act;
            lanes = __popc(act);
            base = -64;  // nothing computed yet
        }
    }
    __device__ static inline double second(double t, double dt, bool half)
    {
        return half ? t + dt / 2 : t + dt;
    }
    template <bool HALF>
    __device__ inline void at(const MemberDev &d, int64_t step, double &h1, double &h2)
    {
        if (d.shape == FIELD_CONSTANT) {
            h1 = a;
            h2 = b;
        } else if (mask) {
            int64_t i = step - 1 - base;
            if (i >= lanes) {
                base = step - 1;
                i = 0;
                const double t = (double)(step + (threadIdx.x & 31)) * d.dt;
                a = f64::field_value(d.shape, t, d.happ, d.fapp);
                b = f64::field_value(d.shape, second(t, d.dt, HALF), d.happ, d.fapp);
            }
            h1 = __shfl_sync(mask, a, (int)i);
            h2 = __shfl_sync(mask, b, (int)i);
        } else {
            const double t = (double)step * d.dt;
            h1 = f64::field_value(d.shape, t, d.happ, d.fapp);
            h2 = f64::field_value(d.shape, second(t, d.dt, HALF), d.happ, d.fapp);
        }
    }
};

// sqrt(sq) > tol for tol > 0 and tol2 = tol * tol, without the root (~600
// cycles) but within a few ulp of equality; comparisons of the bits, as doubles of one
// sign order like integers (an FP64 comparison costs an FP64 instruction).
__device__ inline bool norm_above(double sq, double tol, double tol2)
{
    const int64_t band = 16;  // ulp; sqrt, tol2 and the root's rounding are within 4
    const int64_t inf = 0x7ff0000000000000ll;
    const int64_t s = __double_as_longlong(sq), t = __double_as_longlong(tol2);
    if (s > inf || s < 0) return false;                     // NaN
    if (t > 0x0100000000000000ll && t < 0x7e00000000000000ll) {  // no underflow, no overflow
        if (s > t + band) return true;
        if (s < t - band) return false;
    }
    return sqrt(sq) > tol;
}

// Zero or a magnitude in [2^-80, 2^31): what the pair sum below takes with
// mul_int.  With all of m, r and P in that set, every sum and product of
// P (3 (m.r) r - m) is zero or at least 2^-424 (a sum of numbers that are
// multiples of 2^-k is zero or at least 2^-k) and below 2^160.
__device__ inline bool pair_range(double x)
{
    const uint32_t h = __double2hiint(x) & 0x7fffffffu;
    return h - (943u << 20) < (111u << 20) || (h == 0 && __double2loint(x) == 0);
}

}  // namespace magpy
