// implicit32.cuh -- the FP64 stage map, its FP32 Jacobian and the conversions
// of the mixed-precision implicit midpoint kernels (sllg_fp64.cu on the CUDA
// cores, sllg_tcc.cu on the tensor cores).
#pragma once
#include <cstdint>
#include "mul_int.cuh"

namespace magpy {

// Conversions by integer instructions, the same bits as the hardware's: those
// run on the FP64 pipe (16 cycles of an SM a warp instruction, as FP64 operations on
// one register do; on two they take 19), these take 4-6 cycles of the integer pipes.  Zeros, subnormals,
// infinities and NaN (and numbers past FP32's range) take the hardware's, in a
// call: as predicated instructions those were issued every time (8 of the 54 FP64
// instructions of a particle's iteration).
static __device__ __noinline__ float narrow_any(double x) { return __double2float_rn(x); }
static __device__ __noinline__ double widen_any(float x) { return (double)x; }

__device__ __forceinline__ float narrow(double x)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    if ((hi & 0x7fffffffu) - 0x38100000u >= 0x0fd00000u) return narrow_any(x);
    // exponent and 23 mantissa bits; the 29 below round to nearest even
    const uint32_t m = __funnelshift_l(lo, hi, 3) - 0xc0000000u;
    const uint32_t half = (m & 1u) + 0x7fffffffu;
    uint32_t r;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %2;\n\taddc.u32 %0, %3, 0;\n\t}"
        : "=r"(r)
        : "r"(lo << 3), "r"(half), "r"(m & 0x7fffffffu));
    return __uint_as_float(r | (hi & 0x80000000u));
}

__device__ __forceinline__ double widen(float x)
{
    const uint32_t u = __float_as_uint(x);
    if ((u & 0x7fffffffu) - 0x00800000u >= 0x7f000000u) return widen_any(x);
    return __hiloint2double((int)((((u & 0x7fffffffu) >> 3) + 0x38000000u) | (u & 0x80000000u)),
                            (int)(u << 29));
}

// -(m x v) - alpha m x (m x v): drift and diffusion share this map
// (lib/llg.cpp:14-29, :92-106), linear in v = dt h + sr dwm.
template <class Mul>
__device__ __forceinline__ void stage_map_by(double o[3], const double m[3], double alpha,
                                             const double v[3], Mul mul)
{
    double u[3], w[3];
    u[0] = fma(m[1], v[2], -mul(m[2], v[1]));
    u[1] = fma(m[2], v[0], -mul(m[0], v[2]));
    u[2] = fma(m[0], v[1], -mul(m[1], v[0]));
    w[0] = fma(m[1], u[2], -mul(m[2], u[1]));
    w[1] = fma(m[2], u[0], -mul(m[0], u[2]));
    w[2] = fma(m[0], u[1], -mul(m[1], u[0]));
    for (int c = 0; c < 3; c++) o[c] = fma(-alpha, w[c], -u[c]);
}

struct Double3 { double x, y, z; };

// Any operands (not inlined: rarely used).
static __device__ __noinline__ Double3 stage_map_any(Double3 a, double alpha, Double3 b)
{
    const double m[3] = {a.x, a.y, a.z}, v[3] = {b.x, b.y, b.z};
    double o[3];
    stage_map_by(o, m, alpha, v, [](double x, double y) { return x * y; });
    return Double3{o[0], o[1], o[2]};
}

// Zero or a magnitude in [2^-120, 2^120): mul_int takes every product below (a
// non-zero u, a multiple of 2^-344, is at least that and below 2^241).
__device__ __forceinline__ bool map_range(double x)
{
    const uint32_t h = __double2hiint(x) & 0x7fffffffu;
    return h - (903u << 20) < (240u << 20) || (h | (uint32_t)__double2loint(x)) == 0;
}

// INT: the six plain products on the integer pipes, the same bits.  It pays where
// the FP64 pipe (19 cycles of an SM an instruction) is the bound: 512 members of
// 512 particles on the tensor cores 300 -> 284 us a step.  On the CUDA cores the
// dipolar sum is most of a step and few warps wait for each other: 2.67 -> 2.73 ms
// for a random ensemble of 13 particles, so those keep the FP64 products.
template <bool INT>
__device__ __forceinline__ void stage_map(double o[3], const double m[3], double alpha,
                                          const double v[3])
{
    const auto plain = [](double x, double y) { return x * y; };
    if constexpr (!INT) {
        stage_map_by(o, m, alpha, v, plain);
    } else if (map_range(m[0]) && map_range(m[1]) && map_range(m[2]) && map_range(v[0]) &&
               map_range(v[1]) && map_range(v[2])) {
        stage_map_by(o, m, alpha, v, [](double x, double y) { return mul_int(x, y); });
    } else {
        const Double3 r =
            stage_map_any(Double3{m[0], m[1], m[2]}, alpha, Double3{v[0], v[1], v[2]});
        o[0] = r.x; o[1] = r.y; o[2] = r.z;
    }
}

// J = I - 1/2 d(stage_map)/dm in FP32, with v's own dependence on m through
// the particle's anisotropy (k e e^T, times dt).
__device__ inline void stage_jacobian(float J[9], const float m[3], float alpha, const float v[3],
                                      const float e[3], float dtk)
{
    const float mv = __fmaf_rn(m[2], v[2], __fmaf_rn(m[1], v[1], m[0] * v[0]));
    const float mm = __fmaf_rn(m[2], m[2], __fmaf_rn(m[1], m[1], m[0] * m[0]));
    const float me = __fmaf_rn(m[2], e[2], __fmaf_rn(m[1], e[1], m[0] * e[0]));
    // p = d(map)/dv e = -(m x e) - alpha (m (m.e) - e |m|^2), times dt k
    const float cx[3] = {__fmaf_rn(m[1], e[2], -(m[2] * e[1])), __fmaf_rn(m[2], e[0], -(m[0] * e[2])),
                         __fmaf_rn(m[0], e[1], -(m[1] * e[0]))};
    float p[3];
    for (int c = 0; c < 3; c++)
        p[c] = dtk * __fmaf_rn(alpha, __fmaf_rn(mm, e[c], -(m[c] * me)), -cx[c]);
    // d(map)/dm: [v]_x - alpha ((m.v) I + m v^T - 2 v m^T)
    const float V[9] = {0.f, -v[2], v[1], v[2], 0.f, -v[0], -v[1], v[0], 0.f};
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            float t = __fmaf_rn(m[r], v[c], -2.f * (v[r] * m[c])) + (r == c ? mv : 0.f);
            t = __fmaf_rn(-alpha, t, V[3 * r + c]);
            t = __fmaf_rn(p[r], e[c], t);
            J[3 * r + c] = __fmaf_rn(-0.5f, t, r == c ? 1.f : 0.f);
        }
}

}  // namespace magpy
