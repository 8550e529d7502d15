// sllg_fp64.cu -- the FP64-faithful sLLG ensemble kernel (compiled with
// -fmad=false).
//
// One thread per particle.  A member of n <= 32 particles occupies n
// consecutive lanes of a warp (32/n members per warp) and synchronises with
// __syncwarp on its lane mask; a member of n > 32 particles is one CTA.  The
// member's state stays in registers for the whole run; particles exchange
// their moments through shared memory for the dipolar sum.  Per step the
// kernel follows lib/simulation.cpp:342-405: copy the state, advance the
// step counter, draw 3n increments, take one Heun (lib/integrators.cpp:372)
// or implicit-midpoint (lib/integrators.cpp:576) step at t = step*dt,
// optionally renormalise, and write the zero-order-hold sample.
#include <algorithm>
#include "common.cuh"
#include "fp64_common.cuh"
#include "implicit32.cuh"
#include "llg64.cuh"
#include "plan.hpp"

namespace magpy {
namespace {

struct Particle {
    double ax[3];
    double k, sr, alpha;
    double hj[9];
};

struct Member {
    const MemberDev *d;
    const double *pt, *rt;  // pair tables of the member's cluster
    const float4 *pr;       // FP32 pair table (r0, r1, r2, P), [N][N], index j*n + q
    double *sm;             // [3n] shared moments
    float4 *smf;            // [n] shared FP32 moments (FP32 dipolar sum)
    double *red;            // [p2] shared reduction buffer
    int n, q, p2;
    bool active;
    bool table_ok;          // the particle's pair-table entries allow mul_int
    MemberSync ms;
    // sync(), and whether `ok` holds in every thread of the member
    __device__ inline bool sync_and(bool ok) const
    {
        if (ms.cta) return __syncthreads_and(ok) != 0;
        __syncwarp(ms.mask);
        return __all_sync(ms.mask, ok) != 0;
    }
};

// Shared-memory doubles per member: moments and reduction buffer, or with the
// FP32 dipolar sum FP32 moments (16 bytes a particle) and a reduction buffer
// (one word per warp of a CTA-wide member).
__host__ __device__ inline int slot_doubles(int n, int p2, bool dip32)
{
    return dip32 ? 2 * n + (n > 32 ? 34 : 0) : 3 * n + p2;
}

// Dipolar sum in FP32 from the (r0, r1, r2, P) pair table: fused products,
// FP32 partial sums over 32 sources, added in FP64.  The mixed-precision
// implicit mode uses it inside the FP64 Newton solve.
__device__ inline void dipolar32(const Member &M, double H[3])
{
    const int n = M.n, q = M.q;
    H[0] = H[1] = H[2] = 0.0;
    for (int j0 = 0; j0 < n; j0 += 32) {
        const int j1 = min(n, j0 + 32);
        float h0 = 0.f, h1 = 0.f, h2 = 0.f;
        for (int j = j0; j < j1; j++) {
            const float4 r = __ldg(M.pr + (size_t)j * n + q);  // P = 0 on the diagonal
            const float4 mj = M.smf[j];
            const float d3 = 3.f * __fmaf_rn(mj.z, r.z, __fmaf_rn(mj.y, r.y, __fmul_rn(mj.x, r.x)));
            h0 = __fmaf_rn(r.w, __fmaf_rn(d3, r.x, -mj.x), h0);
            h1 = __fmaf_rn(r.w, __fmaf_rn(d3, r.y, -mj.y), h1);
            h2 = __fmaf_rn(r.w, __fmaf_rn(d3, r.z, -mj.z), h2);
        }
        const double d0 = widen(h0), d1 = widen(h1), d2 = widen(h2);
        H[0] = j0 ? H[0] + d0 : d0;
        H[1] = j0 ? H[1] + d1 : d1;
        H[2] = j0 ? H[2] + d2 : d2;
    }
}

// Effective field of one particle: lib/simulation.cpp:271-290 (anisotropy,
// lib/field.cpp:116-132; Zeeman along z, :81-88; dipolar pair sum, :187-225).
__device__ inline void eff_field(const Member &M, const Particle &pa, double h[3],
                                 const double s[3], double hz)
{
    double dot = s[0] * pa.ax[0] + s[1] * pa.ax[1] + s[2] * pa.ax[2];
    dot *= pa.k;
    h[0] = plus_zero(dot * pa.ax[0]);
    h[1] = plus_zero(dot * pa.ax[1]);
    h[2] = plus_zero(dot * pa.ax[2]) + hz;
    if (M.d->interactions && M.n > 1) {
        if (M.active) {
            M.sm[3 * M.q + 0] = s[0];
            M.sm[3 * M.q + 1] = s[1];
            M.sm[3 * M.q + 2] = s[2];
        }
        const bool ok = M.sync_and(!M.active || (M.table_ok && pair_range(s[0]) &&
                                                 pair_range(s[1]) && pair_range(s[2])));
        const int n = M.n, q = M.q;
        if (M.active && ok) {
            // The same products and sums as below with the products off the
            // FP64 pipe, which bounds the pair sum (18 operations a pair, 10 of
            // them products).  The diagonal's zeros add zero to a sum that is
            // never -0.  512 members of 64, 50 Heun steps: 9.7 -> 6.1 ms (6.2
            // and 6.3 with one or two of the ten left on the FP64 pipe, 6.4
            // with the loop not unrolled or by four).
#pragma unroll 2
            for (int j = 0; j < n; j++) {
                const double mj0 = M.sm[3 * j + 0], mj1 = M.sm[3 * j + 1], mj2 = M.sm[3 * j + 2];
                const double P = __ldg(M.pt + (size_t)j * n + q);
                const double r0 = __ldg(M.rt + ((size_t)0 * n + j) * n + q);
                const double r1 = __ldg(M.rt + ((size_t)1 * n + j) * n + q);
                const double r2 = __ldg(M.rt + ((size_t)2 * n + j) * n + q);
                const double d = mul_int(mj0, r0) + mul_int(mj1, r1) + mul_int(mj2, r2);
                const double t = mul_int(d, 3.0);
                h[0] += mul_int(mul_int(t, r0) - mj0, P);
                h[1] += mul_int(mul_int(t, r1) - mj1, P);
                h[2] += mul_int(mul_int(t, r2) - mj2, P);
            }
        } else if (M.active) {
            for (int j = 0; j < n; j++) {
                if (j == q) continue;
                const double mj0 = M.sm[3 * j + 0], mj1 = M.sm[3 * j + 1], mj2 = M.sm[3 * j + 2];
                const double P = __ldg(M.pt + (size_t)j * n + q);
                const double r0 = __ldg(M.rt + ((size_t)0 * n + j) * n + q);
                const double r1 = __ldg(M.rt + ((size_t)1 * n + j) * n + q);
                const double r2 = __ldg(M.rt + ((size_t)2 * n + j) * n + q);
                const double d = mj0 * r0 + mj1 * r1 + mj2 * r2;
                h[0] += P * (3 * d * r0 - mj0);
                h[1] += P * (3 * d * r1 - mj1);
                h[2] += P * (3 * d * r2 - mj2);
            }
        }
        M.ms.sync();
    }
}

// Square of the member-wide 2-norm with the shim's order: per-particle
// sequential sum of squares, then a pairwise tree over a power-of-two padded
// particle index (the padding's zeros are not added: the partial sums are
// never -0).  The same bits in every thread of the member.
__device__ inline double member_sumsq(const Member &M, const double x[3])
{
    double s = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
    if (!M.ms.cta) {
        if (M.n == 1) return s;
        const int lane = threadIdx.x & 31;
        for (int stride = M.p2 >> 1; stride >= 1; stride >>= 1) {
            const bool add = M.q < stride && M.q + stride < M.n;
            const double o = __shfl_sync(M.ms.mask, s, add ? lane + stride : lane);
            if (add) s = s + o;
        }
        return __shfl_sync(M.ms.mask, s, lane - M.q);
    }
    if (M.active) M.red[M.q] = s;
    M.ms.sync();
    for (int stride = M.p2 / 2; stride >= 1; stride >>= 1) {
        if (M.q < stride && M.q + stride < M.n) M.red[M.q] = M.red[M.q] + M.red[M.q + stride];
        M.ms.sync();
    }
    const double r = M.red[0];
    M.ms.sync();
    return r;
}

__device__ inline bool member_any(const Member &M, bool pred)
{
    if (M.ms.cta) return __syncthreads_or(pred) != 0;
    return __any_sync(M.ms.mask, pred) != 0;
}

// integrator::heun, lib/integrators.cpp:372-405, on the particle's 3x3 block.
__device__ void heun_step(const Member &M, const Particle &pa, double x[3],
                          const double px[3], const double w[3], double hz1, double hz2)
{
    const double dt = M.d->dt, sq = M.d->sqrt_dt;
    double h[3], a[3], b[9], xt[3];
    eff_field(M, pa, h, px, hz1);
    f64::drift(a, px, pa.alpha, h);
    f64::diffusion(b, px, pa.sr, pa.alpha);
    for (int r = 0; r < 3; r++) {
        xt[r] = px[r] + dt * a[r];
        for (int c = 0; c < 3; c++) xt[r] += b[3 * r + c] * w[c] * sq;
    }
    double ta[3], tb[9];
    eff_field(M, pa, h, xt, hz2);
    f64::drift(ta, xt, pa.alpha, h);
    f64::diffusion(tb, xt, pa.sr, pa.alpha);
    for (int r = 0; r < 3; r++) {
        x[r] = px[r] + 0.5 * dt * (ta[r] + a[r]);
        for (int c = 0; c < 3; c++) x[r] += 0.5 * w[c] * sq * (tb[3 * r + c] + b[3 * r + c]);
    }
}

// integrator::implicit_midpoint (lib/integrators.cpp:576-651) with
// optimisation::newton_raphson_noinv (lib/optimisation.cpp:81-149).  The
// Jacobian is block-diagonal (the field Jacobian ignores the dipolar term,
// lib/simulation.cpp:292-303), so the dense dgesv is n independent 3x3
// solves; the convergence norm couples the whole member.
//
// What bounds it: the count of FP64 instructions (64 issue cycles each), 27-40
// iterations a step.  So an iteration is written out with every product and
// sum that llg::drift, llg::diffusion and their Jacobians (llg64.cuh) share
// formed once, in their association, and with multiplications by powers of
// two taken out, which round to the same bits: 0.5 b dwm is b (dwm/2),
// 2 x y + z and d - 0.5 j are one fused operation with an exact product.  The
// applied field is the step's, the root of the norm is avoided (norm_above),
// comparisons are integer: about 335 FP64 instructions an iteration, 470 with
// the functions called one by one (a step of one particle 348 -> 268 us, of 10000
// dimers 0.65 -> 0.47 ms).
__device__ int32_t implicit_step(const Member &M, const Particle &pa, double x[3],
                                 const double px[3], const double w[3], double hz1, double hz2)
{
    const double dt = M.d->dt, sq = M.d->sqrt_dt, Ah = M.d->Ah;
    double hw[3];  // dwm / 2
    double h[3];
    {
        double dwm[3], a[3], b[9];
        for (int c = 0; c < 3; c++) {
            double lo = (w[c] < Ah) ? w[c] : Ah;         // std::min(Ah, dw)
            dwm[c] = ((-Ah < lo) ? lo : -Ah) * sq;       // std::max(-Ah, .) * sqrt(dt)
            hw[c] = 0.5 * dwm[c];
        }
        eff_field(M, pa, h, px, hz1);
        f64::drift(a, px, pa.alpha, h);
        f64::diffusion(b, px, pa.sr, pa.alpha);
        for (int r = 0; r < 3; r++) {
            double g = a[r] * dt;
            for (int c = 0; c < 3; c++) g += b[3 * r + c] * dwm[c];
            x[r] = (g + px[r]) / 2;
        }
    }
    const double tol = M.d->eps * sqrt(member_sumsq(M, x)), tol2 = tol * tol;
    bool going = 2 * tol > tol;  // err starts at 2 tol
    int64_t iter = M.d->max_iter;
    int32_t flag = ST_OK;
    const double hdt = 0.5 * dt, al = pa.alpha, sr = pa.sr, asr = al * sr;
    const double *j = pa.hj;
    while (going && (iter-- > 0)) {
        const double m0 = x[0], m1 = x[1], m2 = x[2];
        eff_field(M, pa, h, x, hz2);
        const double s00 = m0 * m0, s11 = m1 * m1, s22 = m2 * m2;
        const double s12 = s11 + s22, s02 = s00 + s22, s01 = s00 + s11;
        const double p0 = m0 * h[0], p1 = m1 * h[1], p2 = m2 * h[2];
        const double q12 = p1 + p2, q02 = p0 + p2, q01 = p0 + p1;
        const double m2h1 = m2 * h[1], m1h2 = m1 * h[2], m0h2 = m0 * h[2], m2h0 = m2 * h[0],
                     m1h0 = m1 * h[0], m0h1 = m0 * h[1];
        double F[3], J[9];
        {
            // F = x - 0.5 a dt - x0 - 0.5 B dwm
            const double a0 = (m2h1 - m1h2) + al * (h[0] * s12 - m0 * q12);
            const double a1 = (m0h2 - m2h0) + al * (h[1] * s02 - m1 * q02);
            const double a2 = (m1h0 - m0h1) + al * (h[2] * s01 - m2 * q01);
            const double am0 = al * m0, A01 = am0 * m1, A02 = am0 * m2, A12 = al * m1 * m2;
            F[0] = (m0 - a0 * hdt) - px[0];
            F[0] -= (asr * s12) * hw[0];
            F[0] -= (sr * (m2 - A01)) * hw[1];
            F[0] += (sr * (m1 + A02)) * hw[2];
            F[1] = (m1 - a1 * hdt) - px[1];
            F[1] += (sr * (m2 + A01)) * hw[0];
            F[1] -= (asr * s02) * hw[1];
            F[1] -= (sr * (m0 - A12)) * hw[2];
            F[2] = (m2 - a2 * hdt) - px[2];
            F[2] -= (sr * (m1 - A02)) * hw[0];
            F[2] += (sr * (m0 + A12)) * hw[1];
            F[2] -= (asr * s01) * hw[2];
        }
        {
            // drift Jacobian a' (lib/llg.cpp:68-81) into J = I - 0.5 a'
            const double m0j0 = m0 * j[0], m1j0 = m1 * j[0], m2j0 = m2 * j[0];
            const double m0j3 = m0 * j[3], m1j3 = m1 * j[3], m2j3 = m2 * j[3];
            const double m0j6 = m0 * j[6], m1j6 = m1 * j[6], m2j6 = m2 * j[6];
            J[0] = (m2j3 - m1j6) + al * ((s12 * j[0] - q12) - m0 * (m1j3 + m2j6));
            J[3] = ((h[2] - m2j0) + m0j6) +
                   al * (fma(2.0, m0h1, s02 * j[3]) - m1 * ((h[0] + m0j0) + m2j6));
            J[6] = ((m1j0 - h[1]) - m0j3) +
                   al * (fma(2.0, m0h2, s01 * j[6]) - m2 * ((h[0] + m0j0) + m1j3));
            const double m0j1 = m0 * j[1], m1j1 = m1 * j[1], m2j1 = m2 * j[1];
            const double m0j4 = m0 * j[4], m1j4 = m1 * j[4], m2j4 = m2 * j[4];
            const double m0j7 = m0 * j[7], m1j7 = m1 * j[7], m2j7 = m2 * j[7];
            J[1] = ((m2j4 - h[2]) - m1j7) +
                   al * (fma(2.0, m1h0, s12 * j[1]) - m0 * ((h[1] + m1j4) + m2j7));
            J[4] = (m0j7 - m2j1) + al * ((s02 * j[4] - q02) - m1 * (m0j1 + m2j7));
            J[7] = ((h[0] + m1j1) - m0j4) +
                   al * (fma(2.0, m1h2, s01 * j[7]) - m2 * ((h[1] + m0j1) + m1j4));
            const double m0j2 = m0 * j[2], m1j2 = m1 * j[2], m2j2 = m2 * j[2];
            const double m0j5 = m0 * j[5], m1j5 = m1 * j[5], m2j5 = m2 * j[5];
            const double m0j8 = m0 * j[8], m1j8 = m1 * j[8], m2j8 = m2 * j[8];
            J[2] = ((h[1] + m2j5) - m1j8) +
                   al * (fma(2.0, m2h0, s12 * j[2]) - m0 * ((h[2] + m1j5) + m2j8));
            J[5] = ((-h[0] - m2j2) + m0j8) +
                   al * (fma(2.0, m2h1, s02 * j[5]) - m1 * ((h[2] + m0j2) + m2j8));
            J[8] = (m1j2 - m0j5) + al * ((s01 * j[8] - q01) - m2 * (m0j2 + m1j5));
            for (int k = 0; k < 9; k++) J[k] = fma(-0.5, J[k], k % 4 == 0 ? 1.0 : 0.0);
        }
        {
            // - 0.5 b'_k dwm_k (lib/llg.cpp:118-158), k = 0, 1, 2 in turn: b' has
            // the entries +-sr, -asr m, 2 asr m and 0 (whose zero products
            // change nothing: an entry of J is never -0)
            const double c0 = asr * m0, c1 = asr * m1, c2 = asr * m2;
            const double p00 = c0 * hw[0], p01 = c0 * hw[1], p02 = c0 * hw[2];
            const double p10 = c1 * hw[0], p11 = c1 * hw[1], p12 = c1 * hw[2];
            const double p20 = c2 * hw[0], p21 = c2 * hw[1], p22 = c2 * hw[2];
            const double t0 = sr * hw[0], t1 = sr * hw[1], t2 = sr * hw[2];
            J[0] = (J[0] + p11) + p22;
            J[1] = (fma(-2.0, p10, J[1]) + p21) + t2;
            J[2] = (fma(-2.0, p20, J[2]) - t1) + p02;
            J[3] = fma(-2.0, p01, J[3] + p10) - t2;
            J[4] = (J[4] + p00) + p22;
            J[5] = fma(-2.0, p21, J[5] + t0) + p12;
            J[6] = fma(-2.0, p02, (J[6] + p20) + t1);
            J[7] = fma(-2.0, p22, (J[7] - t0) + p21);
            J[8] = (J[8] + p00) + p11;
        }
        double sol[3] = {-F[0], -F[1], -F[2]};
        int info = M.active ? f64::solve3_bits(J, sol) : 0;
        if (member_any(M, info != 0)) {
            flag = ST_SINGULAR;
            x[0] = -F[0]; x[1] = -F[1]; x[2] = -F[2];
            break;
        }
        going = norm_above(member_sumsq(M, sol), tol, tol2);
        x[0] = sol[0] + m0;
        x[1] = sol[1] + m1;
        x[2] = sol[2] + m2;
    }
    if (flag == ST_OK && iter == -1) flag = ST_NEWTON_MAXITER;
    for (int r = 0; r < 3; r++) x[r] = 2 * x[r] - px[r];
    return flag;
}

// ---- implicit midpoint of the mixed-precision mode ----
// The equation, its FP64 residual and state, the tolerance (eps times the norm
// of the reference's first iterate) and the stopping test (|dx| <= tol over
// the member, at most max_iter iterations) are those of implicit_step; the
// dipolar sum is FP32 (dipolar32), and the iteration is steered by the
// equation's own Jacobian instead of the reference's: that one writes the
// drift term without dt (lib/integrators.cpp:633) and reads another
// particle's block of the field Jacobian (lib/llg.cpp:386), contracts by
// about one half per iteration and takes 27-40 of them a step, this one by
// dt |D| (the dipolar coupling is left out of it) and takes 3.  FP64 costs 64
// issue cycles a warp instruction here, so the step's length is the count of
// its FP64 operations: iterations times ~60.  700 members of 13 particles, dt =
// 2e-13: 20 steps 4.38 ms with the reference's iteration, 0.31 ms with this one.

// Member-wide FP32 sum, the same bits in every thread of the member.
__device__ inline float member_sum32(const Member &M, float v)
{
    if (!M.ms.cta) {
        const int lane = threadIdx.x & 31, first = lane - M.q;
        for (int stride = M.p2 >> 1; stride >= 1; stride >>= 1) {
            const float o = __shfl_sync(M.ms.mask, v, M.q + stride < M.n ? lane + stride : lane);
            if (M.q + stride < M.n && M.q < stride) v += o;
        }
        return __shfl_sync(M.ms.mask, v, first);
    }
    float *red = (float *)M.red;
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w];
    __syncthreads();
    return s;
}
__device__ inline double member_sum64(const Member &M, double v)
{
    if (!M.ms.cta) {
        const int lane = threadIdx.x & 31, first = lane - M.q;
        for (int stride = M.p2 >> 1; stride >= 1; stride >>= 1) {
            const double o = __shfl_sync(M.ms.mask, v, M.q + stride < M.n ? lane + stride : lane);
            if (M.q + stride < M.n && M.q < stride) v += o;
        }
        return __shfl_sync(M.ms.mask, v, first);
    }
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0) M.red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += M.red[w];
    __syncthreads();
    return s;
}

// Stage increment dt a + B dwm at the state s, and its v.
__device__ inline void stage32(const Member &M, const Particle &pa, const double s[3], double hz,
                               const double sdw[3], double dt, double g[3], double v[3])
{
    double H[3] = {0.0, 0.0, 0.0};
    if (M.d->interactions && M.n > 1) {
        if (M.active) M.smf[M.q] = make_float4(narrow(s[0]), narrow(s[1]), narrow(s[2]), 0.f);
        M.ms.sync();
        if (M.active) dipolar32(M, H);
        M.ms.sync();
    }
    const double dot = pa.k * fma(s[2], pa.ax[2], fma(s[1], pa.ax[1], s[0] * pa.ax[0]));
    v[0] = fma(dt, fma(dot, pa.ax[0], H[0]), sdw[0]);
    v[1] = fma(dt, fma(dot, pa.ax[1], H[1]), sdw[1]);
    v[2] = fma(dt, fma(dot, pa.ax[2], H[2] + hz), sdw[2]);
    stage_map<false>(g, s, pa.alpha, v);
}

__device__ int32_t implicit_step32(const Member &M, const Particle &pa, double x[3],
                                   const double px[3], const double w[3], double hz1, double hz2)
{
    const MemberDev &d = *M.d;
    const double dt = d.dt, sq = d.sqrt_dt, Ah = d.Ah;
    double sdw[3], g[3], v[3];
    for (int c = 0; c < 3; c++) {
        const double lo = (w[c] < Ah) ? w[c] : Ah;       // std::min(Ah, dw)
        sdw[c] = pa.sr * (((-Ah < lo) ? lo : -Ah) * sq);  // std::max(-Ah, .) * sqrt(dt)
    }
    stage32(M, pa, px, hz1, sdw, dt, g, v);
    // the reference's first iterate (g + x0)/2 sets the tolerance; the
    // iteration starts from the explicit midpoint x0 + g/2, whose error is of
    // second order in the step
    double s2 = 0.0;
    for (int c = 0; c < 3; c++) {
        const double r = 0.5 * (g[c] + px[c]);
        s2 = fma(r, r, s2);
        x[c] = fma(0.5, g[c], px[c]);
    }
    s2 = member_sum64(M, M.active ? s2 : 0.0);
    const double tol2 = d.eps * d.eps * s2;
    // FP32 bounds that decide the stopping test but for a narrow band, in
    // which (and where FP32 could underflow) the FP64 norm is formed
    const float far = (float)(tol2 * 1.0001), near = (float)(tol2 * 0.9999);
    const bool fp32_ok = near > 1e-30f;
    int64_t iter = d.max_iter;
    int32_t flag = ST_OK;
    // err starts at 2 tol, as in the reference: no iteration for a tolerance
    // of zero, below zero, infinite or NaN
    bool going = d.eps > 0 && s2 > 0 && s2 < INFINITY;
    if (!going)  // the result is the reference's first iterate
        for (int c = 0; c < 3; c++) x[c] = fma(-0.5, px[c], x[c]);
    const float ef[3] = {(float)pa.ax[0], (float)pa.ax[1], (float)pa.ax[2]};
    const float dtk = (float)(dt * pa.k), alf = (float)pa.alpha;
    while (going && (iter-- > 0)) {
        stage32(M, pa, x, hz2, sdw, dt, g, v);
        // F = x - x0 - g/2 (lib/integrators.cpp:621-627), and J sol = -F
        double mF[3];
        float sol[3], J[9];
        for (int c = 0; c < 3; c++) {
            mF[c] = fma(0.5, g[c], px[c]) - x[c];
            sol[c] = narrow(mF[c]);
        }
        const float mf[3] = {narrow(x[0]), narrow(x[1]), narrow(x[2])};
        const float vf[3] = {narrow(v[0]), narrow(v[1]), narrow(v[2])};
        stage_jacobian(J, mf, alf, vf, ef, dtk);
        const int info = M.active ? f64::solve3<float>(J, sol) : 0;
        if (member_any(M, info != 0)) {  // as implicit_step: x = -F is the result
            for (int c = 0; c < 3; c++) x[c] = mF[c];
            flag = ST_SINGULAR;
            break;
        }
        float e32 = __fmaf_rn(sol[2], sol[2], __fmaf_rn(sol[1], sol[1], sol[0] * sol[0]));
        e32 = member_sum32(M, M.active ? e32 : 0.f);
        if (fp32_ok && e32 > far) {
            going = true;
        } else if (fp32_ok && e32 < near) {
            going = false;
        } else {
            double e2 = 0.0;
            for (int c = 0; c < 3; c++) e2 = fma((double)sol[c], (double)sol[c], e2);
            e2 = member_sum64(M, M.active ? e2 : 0.0);
            going = e2 > tol2;
        }
        for (int c = 0; c < 3; c++) x[c] += widen(sol[c]);
    }
    if (flag == ST_OK && iter == -1) flag = ST_NEWTON_MAXITER;
    for (int c = 0; c < 3; c++) x[c] = 2 * x[c] - px[c];
    return flag;
}

// MAXT: the largest CTA of the instantiation (256 for warp-packed members,
// 512 or 1024 for one member per CTA), so that the register budget of a
// thread never exceeds what a full CTA may use.
template <bool IMPLICIT, bool DIP32, int MAXT>
__global__ void __launch_bounds__(MAXT) sllg_fp64_kernel(DevPlan p)
{
    extern __shared__ __align__(16) double smem[];
    const int n = p.n;
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    const int slot_size = slot_doubles(n, p2, DIP32);

    Member M;
    int64_t e;
    if (n > 32) {
        e = blockIdx.x;
        M.q = threadIdx.x;
        M.active = M.q < n;
        M.ms.cta = true;
        M.ms.mask = 0xffffffffu;
        M.sm = smem;
    } else {
        const int mpw = (p.members_per_warp > 0 && p.members_per_warp < 32 / n) ? p.members_per_warp : 32 / n;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int sub = lane / n;
        const int slot = warp * mpw + sub;
        e = (int64_t)blockIdx.x * ((blockDim.x >> 5) * mpw) + slot;
        if (sub >= mpw || e >= p.E) return;  // whole member leaves together
        M.q = lane % n;
        M.active = true;
        M.ms.cta = false;
        M.ms.mask = (n == 32) ? 0xffffffffu : (((1u << n) - 1u) << (sub * n));
        M.sm = smem + (size_t)slot * slot_size;
    }
    // FP64: moments then the reduction buffer; FP32 dipolar sum: float4
    // moments (16-byte aligned: 2n doubles a member) then the buffer
    M.red = M.sm + (DIP32 ? 2 * n : 3 * n);
    M.smf = (float4 *)M.sm;
    M.n = n;
    M.p2 = p2;
    const MemberDev *md = p.members + e;
    M.d = md;
    M.pt = p.pt + md->cluster_off;
    M.rt = p.rt + 3 * md->cluster_off;
    M.pr = DIP32 ? p.pr + md->cluster_off : nullptr;
    M.table_ok = true;
    if (!DIP32 && md->interactions && n > 1 && M.active)
        for (int j = 0; j < n; j++)
            M.table_ok &= pair_range(__ldg(M.pt + (size_t)j * n + M.q)) &&
                          pair_range(__ldg(M.rt + ((size_t)0 * n + j) * n + M.q)) &&
                          pair_range(__ldg(M.rt + ((size_t)1 * n + j) * n + M.q)) &&
                          pair_range(__ldg(M.rt + ((size_t)2 * n + j) * n + M.q));

    const int64_t P = p.P;
    const int64_t g = md->pbase + (M.active ? M.q : 0);
    Particle pa;
    double x[3], px[3];
    for (int c = 0; c < 3; c++) {
        pa.ax[c] = p.axes[c * P + g];
        x[c] = p.m0[c * P + g];
        px[c] = x[c];
    }
    pa.k = p.k_red[g];
    pa.sr = p.sr[g];
    pa.alpha = md->alpha;
    if (IMPLICIT && !DIP32)
        for (int k = 0; k < 9; k++) pa.hj[k] = p.hj[k * P + g];
    const double scale = p.out_scale[e];
    const int64_t S = p.S;
    const int64_t *sched = p.sched + md->sched_off;
    const double *noise = p.noise ? p.noise + md->noise_off : nullptr;
    const int64_t per_step = 3 * (int64_t)n;

    if (M.active && p.mx) {  // sample 0: the initial state, simulation.cpp:212-219
        p.mx[g] = x[0] * scale;
        p.my[g] = x[1] * scale;
        p.mz[g] = x[2] * scale;
    }
    // lanes of a warp share the applied field where their members take the
    // same steps through the same waveform
    AppliedField af;
    {
        const unsigned act = __activemask();
        const MemberDev *d0 = p.members + __shfl_sync(act, e, __ffs(act) - 1);
        af.init(*md, __all_sync(act, md->dt == d0->dt && md->happ == d0->happ &&
                                         md->fapp == d0->fapp && md->shape == d0->shape &&
                                         md->sched_off == d0->sched_off &&
                                         md->noise_len == d0->noise_len));
    }
    int32_t status = ST_OK;
    uint64_t step = 0;
    int64_t s = 1;
    for (; s < S; s++) {
        const int64_t ks = sched[s];
        while ((int64_t)step < ks) {
            px[0] = x[0]; px[1] = x[1]; px[2] = x[2];
            step++;
            double hz1, hz2;
            double w[3];
            if (noise) {
                if ((int64_t)step * per_step > md->noise_len) {
                    status |= ST_NOISE_EXHAUSTED;
                    step--;
                    goto finished;
                }
                const double *wp = noise + (int64_t)(step - 1) * per_step + 3 * M.q;
                w[0] = wp[0]; w[1] = wp[1]; w[2] = wp[2];
            } else {
                Normals4 r = wiener_normals(md->seed, step, (uint32_t)M.q);
                w[0] = r.a; w[1] = r.b; w[2] = r.c;
            }
            af.at<IMPLICIT>(*md, (int64_t)step, hz1, hz2);
            if (DIP32) status |= implicit_step32(M, pa, x, px, w, hz1, hz2);
            else if (IMPLICIT) status |= implicit_step(M, pa, x, px, w, hz1, hz2);
            else heun_step(M, pa, x, px, w, hz1, hz2);
            if (md->renorm) {  // simulation.cpp:379-387
                double s2 = 0.0;
                s2 = s2 + x[0] * x[0];
                s2 = s2 + x[1] * x[1];
                s2 = s2 + x[2] * x[2];
                const double norm = sqrt(s2);
                for (int c = 0; c < 3; c++) x[c] = x[c] / norm;
            }
        }
        if (M.active && p.mx) {  // zero-order hold, simulation.cpp:398-405
            const int64_t o = s * P + g;
            p.mx[o] = px[0] * scale;
            p.my[o] = px[1] * scale;
            p.mz[o] = px[2] * scale;
        }
    }
finished:
    if (M.active && p.mx)  // samples a stopped member never reached
        for (; s < S; s++) {
            const int64_t o = s * P + g;
            p.mx[o] = NAN; p.my[o] = NAN; p.mz[o] = NAN;
        }
    bool bad = M.active && !(isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]));
    if (member_any(M, bad)) status |= ST_NONFINITE;
    if (M.q == 0) {
        if (p.status) p.status[e] = status;
        if (p.steps) p.steps[e] = (int64_t)step;
    }
}

}  // namespace

cudaError_t launch_fp64(const DevPlan &p, cudaStream_t stream)
{
    if (p.E == 0) return cudaSuccess;
    const int n = p.n;
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    // the mixed-precision implicit mode: FP64 Newton, FP32 dipolar sum
    const bool dip32 = p.use_implicit && p.pr != nullptr;
    if (!dip32 && fp64_lanes_fit(p)) return launch_fp64_lanes(p, stream);
    const size_t slot = (size_t)slot_doubles(n, p2, dip32) * sizeof(double);
    dim3 grid, block;
    size_t shmem;
    DevPlan q = p;  // with the members per warp filled in
    if (n > 32) {
        block = dim3(((n + 31) / 32) * 32);
        grid = dim3((unsigned)p.E);
        shmem = slot;
    } else {
        int mpw = (p.members_per_warp > 0 && p.members_per_warp < 32 / n) ? p.members_per_warp : 32 / n;
        int warps = p.block_warps;
        if (warps <= 0) {
            // An FP64 warp instruction takes 64 cycles of its sub-partition
            // however many lanes are active, and one warp fills that pipe: an
            // ensemble that needs fewer warps than the chip has
            // sub-partitions is spread over them one warp each (700 members of
            // 13 particles, implicit: 350 warps in 88 CTAs of four warps keep
            // 64 SMs idle), members apart where that costs no second warp.
            // 10000 dimers, 10 implicit steps: 6.5 ms in CTAs of four warps (five
            // SMs take a second CTA), 4.7 ms in CTAs of one.
            const int64_t subs = sub_partitions();
            if (p.members_per_warp <= 0)
                mpw = (int)std::min<int64_t>(32 / n, std::max<int64_t>(1, (p.E + subs - 1) / subs));
            warps = (p.E + mpw - 1) / mpw <= 4 * subs ? 1 : 4;
        }
        q.members_per_warp = mpw;
        block = dim3(32 * warps);
        const int64_t per_block = (int64_t)warps * mpw;
        grid = dim3((unsigned)((p.E + per_block - 1) / per_block));
        shmem = slot * per_block;
    }
    const unsigned bt = block.x;
    if (p.use_implicit && dip32) {
        if (bt <= 256) sllg_fp64_kernel<true, true, 256><<<grid, block, shmem, stream>>>(q);
        else if (bt <= 512) sllg_fp64_kernel<true, true, 512><<<grid, block, shmem, stream>>>(q);
        else sllg_fp64_kernel<true, true, 1024><<<grid, block, shmem, stream>>>(q);
    } else if (p.use_implicit) {
        if (bt <= 256) sllg_fp64_kernel<true, false, 256><<<grid, block, shmem, stream>>>(q);
        else if (bt <= 512) sllg_fp64_kernel<true, false, 512><<<grid, block, shmem, stream>>>(q);
        else sllg_fp64_kernel<true, false, 1024><<<grid, block, shmem, stream>>>(q);
    } else {
        if (bt <= 256) sllg_fp64_kernel<false, false, 256><<<grid, block, shmem, stream>>>(q);
        else if (bt <= 512) sllg_fp64_kernel<false, false, 512><<<grid, block, shmem, stream>>>(q);
        else sllg_fp64_kernel<false, false, 1024><<<grid, block, shmem, stream>>>(q);
    }
    return cudaGetLastError();
}

// ---- component evaluation (device versions of the pinned functions) ----
namespace {
__global__ void components_kernel(int64_t n, const double *m, const double *h,
                                  const double *hj, const double *axis, const double *alpha,
                                  const double *sr, double *drift, double *diffusion,
                                  double *drift_jac, double *diff_jac, double *anis)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double mm[3] = {m[3 * i], m[3 * i + 1], m[3 * i + 2]};
    double hh[3] = {h[3 * i], h[3 * i + 1], h[3 * i + 2]};
    if (drift) {
        double d[3];
        f64::drift(d, mm, alpha[i], hh);
        for (int c = 0; c < 3; c++) drift[3 * i + c] = d[c];
    }
    if (diffusion) {
        double b[9];
        f64::diffusion(b, mm, sr[i], alpha[i]);
        for (int c = 0; c < 9; c++) diffusion[9 * i + c] = b[c];
    }
    if (drift_jac) {
        double hjj[9], j[9];
        for (int c = 0; c < 9; c++) hjj[c] = hj[9 * i + c];
        f64::drift_jacobian(j, mm, alpha[i], hh, hjj);
        for (int c = 0; c < 9; c++) drift_jac[9 * i + c] = j[c];
    }
    if (diff_jac) {
        double j[27];
        f64::diffusion_jacobian(j, mm, sr[i], alpha[i]);
        for (int c = 0; c < 27; c++) diff_jac[27 * i + c] = j[c];
    }
    if (anis) {
        double ax[3] = {axis[3 * i], axis[3 * i + 1], axis[3 * i + 2]}, hh2[3];
        f64::uniaxial(hh2, mm, ax);
        for (int c = 0; c < 3; c++) anis[3 * i + c] = hh2[c];
    }
}
}  // namespace

cudaError_t launch_components(int64_t n, const double *m, const double *h, const double *hj,
                              const double *axis, const double *alpha, const double *sr,
                              double *drift, double *diffusion, double *drift_jac,
                              double *diff_jac, double *anis, cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    components_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(
        n, m, h, hj, axis, alpha, sr, drift, diffusion, drift_jac, diff_jac, anis);
    return cudaGetLastError();
}

}  // namespace magpy
