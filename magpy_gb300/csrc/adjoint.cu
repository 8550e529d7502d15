// adjoint.cu -- pathwise adjoint of the stochastic Heun step over fixed noise.
//
// Forward map of one step (reduced units, per particle, with the increments w
// of the step fixed by the counter-based generator):
//     h(x)  = k (x.e) e + D x + happ s(t) z          (lib/simulation.cpp:271-290)
//     v     = dt h + sqrt(dt) sr w
//     F(m,v)= -(m x v) - alpha (m (m.v) - v |m|^2)    (drift and diffusion of
//             lib/llg.cpp:14-106 share this form, linear in v)
//     x~    = x + F(x, v1(x)),   x' = x + (F(x, v1(x)) + F(x~, v2(x~))) / 2
// (the Stratonovich Heun step of lib/integrators.cpp:372-405).
//
// Reverse step, for the adjoint lambda' = dJ/dx':
//     g2 = lambda'/2,  mu2 = M(x~)^T g2,  eta2 = dt mu2
//     lam~ = J_m(x~,v2)^T g2 + (A + D)^T eta2
//     g1 = lambda'/2 + lam~,  mu1 = M(x)^T g1,  eta1 = dt mu1
//     lambda = lambda' + lam~ + J_m(x,v1)^T g1 + (A + D)^T eta1
// with M(m)^T u = m x u - alpha (m (m.u) - u |m|^2),
//      J_m(m,v)^T u = u x v - alpha ((m.v) u + (m.u) v - 2 (u.v) m),
//      A = k e e^T (symmetric), D^T = V D V^-1 (V = diag of reduced volumes,
//      so the forward pair table serves the transpose too).
// Parameter sensitivities accumulated along the way:
//     Gh = sum mu.h (d/d dt), Gw = sum mu.(sr w) (d/d sqrt(dt)),
//     Ga = sum g.dF/dalpha, Ghapp = sum eta_z s, Gc = sum eta.(D x)/c.
// The forward pass keeps every step's moments and dipolar fields where they fit
// (adjoint_keep in rules.hpp); otherwise checkpoints every C steps keep the
// float-float state, and each segment is recomputed forward (same code, same bits)
// into a buffer of moments (and fields) and then swept backward.
//
// What bounds it: the dipolar sums, by their instructions, table reads and
// chains.  In a large ensemble a thread integrates particle q of two members
// (they share the cluster), in packed FP32 instructions on (member A, member B)
// pairs: each table entry read and each instruction of a sum serves both.  The
// dipolar fields are kept beside the moments, so that a step takes four sums in
// all (two forward, two of the adjoint), six where a segment is recomputed, eight
// without kept fields.  27 particles, 2048 members, 512 steps with the host's
// copies: 8.4 -> 5.4 ms with a segment's fields kept, 3.9 with the run's.
#include "common.cuh"
#include "llg32.cuh"
#include "plan.hpp"

namespace magpy {
namespace {

// The sweep's arithmetic on one member a thread (V = float) or on two (float2),
// with the same roundings: no contraction but the written one.
using magpy::mul2;
using magpy::add2;
using magpy::fma2;
using magpy::neg2;
__device__ inline float mul2(float a, float b) { return __fmul_rn(a, b); }
__device__ inline float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ inline float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ inline float neg2(float a) { return -a; }
template <class V> __device__ inline V all(float a);
template <> __device__ inline float all<float>(float a) { return a; }
template <> __device__ inline float2 all<float2>(float a) { return make_float2(a, a); }
template <class V> __device__ inline V both(float a, float b);
template <> __device__ inline float both<float>(float a, float) { return a; }
template <> __device__ inline float2 both<float2>(float a, float b) { return make_float2(a, b); }
__device__ inline float first(float a) { return a; }
__device__ inline float first(float2 a) { return a.x; }
__device__ inline float last(float a) { return a; }
__device__ inline float last(float2 a) { return a.y; }
template <class V> constexpr int WIDTH = sizeof(V) / sizeof(float);

template <class V> __device__ inline V dot3(const V a[3], const V b[3])
{
    return fma2(a[2], b[2], fma2(a[1], b[1], mul2(a[0], b[0])));
}

// a x b, one component
template <class V> __device__ inline V cross(const V a[3], const V b[3], int i, int j)
{
    return fma2(a[i], b[j], neg2(mul2(a[j], b[i])));
}

// F(m, v)
template <class V> __device__ inline void llg(V o[3], const V m[3], V alpha, const V v[3])
{
    const V mv = dot3(m, v), mm = dot3(m, m);
    const V c[3] = {cross(m, v, 1, 2), cross(m, v, 2, 0), cross(m, v, 0, 1)};
    for (int i = 0; i < 3; i++)
        o[i] = fma2(alpha, fma2(v[i], mm, neg2(mul2(m[i], mv))), neg2(c[i]));
}

// (hi, lo) + d, the float-float state
template <class V> __device__ inline void dd_add(V &hi, V &lo, V d)
{
    const V y = add2(d, lo);
    const V s = add2(hi, y);
    const V bb = add2(s, neg2(hi));
    lo = add2(add2(hi, neg2(add2(s, neg2(bb)))), add2(y, neg2(bb)));
    hi = s;
}

// M(m)^T u
template <class V> __device__ inline void MT(V o[3], const V m[3], V alpha, const V u[3])
{
    const V mu = dot3(m, u), mm = dot3(m, m), na = neg2(alpha);
    const V c[3] = {cross(m, u, 1, 2), cross(m, u, 2, 0), cross(m, u, 0, 1)};
    for (int i = 0; i < 3; i++) o[i] = fma2(na, fma2(m[i], mu, neg2(mul2(u[i], mm))), c[i]);
}

// J_m(m, v)^T u, accumulated into o
template <class V>
__device__ inline void JmT_add(V o[3], const V m[3], V alpha, const V v[3], const V u[3])
{
    const V mv = dot3(m, v), mu = dot3(m, u), na = neg2(alpha);
    const V uv2 = mul2(all<V>(-2.f), dot3(u, v));
    const V c[3] = {cross(u, v, 1, 2), cross(u, v, 2, 0), cross(u, v, 0, 1)};
    for (int i = 0; i < 3; i++)
        o[i] = add2(o[i], fma2(na, fma2(uv2, m[i], fma2(mu, v[i], mul2(mv, u[i]))), c[i]));
}

// u . dF/dalpha
template <class V> __device__ inline V dFda(const V m[3], const V v[3], const V u[3])
{
    return neg2(fma2(dot3(m, u), dot3(m, v), neg2(mul2(dot3(u, v), dot3(m, m)))));
}

// Particle q of the member e (V = float) or of e and e + 1 (V; where there
// is no second one, its half repeats the first's, and nothing of it is written
// or summed).
template <class V> struct AdjMember {
    int n, q;
    bool active, second;
    MemberSync ms;
    float4 *xy;           // [n] exchange buffer: x, y, z or x, x', y, y'
    float2 *zz;           // [n] z, z' (float2)
    const float4 *pr;     // pair table (r0, r1, r2, P), index j*n + q
    // SPLIT: this warp's share of the sources, and the exchange of partial sums
    // ([2 buffers][2 warps][3][32])
    int half, j0, j1;
    V *part;
    bool writes;          // this thread writes results (active, first warp)
    V ax[3], k, srq, vq;
    uint64_t seed[2];
    int64_t e, g;         // first member, its global particle index
    int64_t pair, pairs;  // the particle's index in the internal buffers, their size
    V *buffers;      // SPLIT: both exchange buffers
    __device__ inline V *half_buffer(V *now) const
    {
        return now == buffers ? buffers + 192 : buffers;
    }
};

__device__ inline void put(const AdjMember<float> &M, int q, const float s[3])
{
    M.xy[q] = make_float4(s[0], s[1], s[2], 0.f);
}
__device__ inline void put(const AdjMember<float2> &M, int q, const float2 s[3])
{
    M.xy[q] = make_float4(s[0].x, s[0].y, s[1].x, s[1].y);
    M.zz[q] = s[2];
}
__device__ inline void get(const AdjMember<float> &M, int j, float m[3])
{
    const float4 v = M.xy[j];
    m[0] = v.x;
    m[1] = v.y;
    m[2] = v.z;
}
__device__ inline void get(const AdjMember<float2> &M, int j, float2 m[3])
{
    const float4 v = M.xy[j];
    m[0] = make_float2(v.x, v.y);
    m[1] = make_float2(v.z, v.w);
    m[2] = M.zz[j];
}

// sum_j P_qj (3 r_qj (r_qj . s_j) - s_j): the dipolar field of the moments s.
// SPLIT: two warps hold the same members and sum over half of the sources
// each; both add the halves in the same order.
template <bool SPLIT, class V>
__device__ inline void dip(AdjMember<V> &M, const V s[3], V out[3])
{
    out[0] = out[1] = out[2] = all<V>(0.f);
    if (M.n < 2) return;
    if (M.active) put(M, M.q, s);
    M.ms.sync();
    if (M.active)
#pragma unroll 9
        for (int j = SPLIT ? M.j0 : 0; j < (SPLIT ? M.j1 : M.n); j++) {
            const float4 r = __ldg(M.pr + (size_t)j * M.n + M.q);  // P = 0 on the diagonal
            const V rx = all<V>(r.x), ry = all<V>(r.y), rz = all<V>(r.z), rw = all<V>(r.w);
            V m[3];
            get(M, j, m);
            const V d3 =
                mul2(all<V>(3.f), fma2(m[2], rz, fma2(m[1], ry, mul2(m[0], rx))));
            out[0] = fma2(rw, fma2(d3, rx, neg2(m[0])), out[0]);
            out[1] = fma2(rw, fma2(d3, ry, neg2(m[1])), out[1]);
            out[2] = fma2(rw, fma2(d3, rz, neg2(m[2])), out[2]);
        }
    if (SPLIT) {
        const int lane = threadIdx.x & 31;
        for (int c = 0; c < 3; c++) M.part[(3 * M.half + c) * 32 + lane] = out[c];
        __syncthreads();
        for (int c = 0; c < 3; c++)
            out[c] = add2(M.part[c * 32 + lane], M.part[(3 + c) * 32 + lane]);
        // the other buffer next: no warp is two sums ahead of the other
        M.part = M.half_buffer(M.part);
    } else {
        M.ms.sync();
    }
}

struct AdjArgs {
    int64_t E, P, S, K;
    int n, C, interactions;
    const MemberDev *members;
    const double *m0, *axes, *k_red, *sr, *v_red;
    const float4 *pr;
    const float2 *stab;   // sin of the applied waveform at t_k and t_k + dt, per step
    float happ, dt, sq, alpha, c;
    const int64_t *sched;
    float *ck;            // [K/C + 1][6][pairs] V: checkpoints (hi xyz, lo xyz); none if `whole`
    // [C][3 or 9][pairs] V: moments (and dipolar fields) of the segment being
    // swept; `whole`: [K][9][pairs] of the whole run, written by the forward pass
    float *seg;
    bool whole;
    const double *out_scale; // [E] Ms
    double *mx, *my, *mz; // samples [S][P]
    const double *wz;     // [S] dJ/d(reduced m_z of any particle at sample s)
    double *grad;         // [5] Gh, Gw, Ga, Ghapp, Gc
    int32_t *status;
};

template <bool SPLIT, class V>
__device__ inline bool setup_member(const AdjArgs &A, AdjMember<V> &M, float4 *smem)
{
    const int n = A.n;
    constexpr int W = WIDTH<V>;
    int64_t two;  // index of the thread's members
    int slot = 0, slots = 1;
    if (n > 32) {
        two = blockIdx.x;
        M.q = threadIdx.x;
        M.active = M.q < n;
        M.ms.cta = true;
        M.ms.mask = 0xffffffffu;
    } else {
        const int mpw = 32 / n;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / n;
        slots = (blockDim.x >> 5) * mpw;
        slot = warp * mpw + sub;
        two = SPLIT ? (int64_t)blockIdx.x * mpw + sub : (int64_t)blockIdx.x * slots + slot;
        if (sub >= mpw || W * two >= A.E) return false;
        M.q = lane % n;
        M.active = true;
        M.ms.cta = false;
        M.ms.mask = (n == 32) ? 0xffffffffu : (((1u << n) - 1u) << (sub * n));
    }
    M.xy = smem + (size_t)slot * n;
    M.zz = (float2 *)(smem + (size_t)slots * n) + (size_t)slot * n;
    M.n = n;
    M.pr = A.pr;
    M.half = SPLIT ? (int)(threadIdx.x >> 5) : 0;
    M.j0 = M.half ? n / 2 : 0;
    M.j1 = SPLIT && !M.half ? n / 2 : n;
    M.buffers = (V *)(smem + (size_t)slots * n + (size_t)(slots * n + 1) / 2);
    M.part = M.buffers;
    M.writes = M.active && M.half == 0;
    M.e = W * two;
    M.second = W == 2 && M.e + 1 < A.E;
    const int q = M.active ? M.q : 0;
    M.g = M.e * n + q;
    M.pair = two * n + q;
    M.pairs = (A.E + W - 1) / W * n;
    for (int c = 0; c < 3; c++) M.ax[c] = all<V>((float)A.axes[c * A.P + M.g]);
    M.k = all<V>((float)A.k_red[M.g]);
    M.srq = all<V>((float)A.sr[M.g]);
    M.vq = all<V>((float)A.v_red[M.g]);
    M.seed[0] = A.members[M.e].seed;
    M.seed[1] = A.members[M.e + (M.second ? 1 : 0)].seed;
    return true;
}

// The increments of the particle at step k.
template <class V> __device__ inline void increments(const AdjMember<V> &M, int64_t k, V w[3])
{
    const Normals4 a = wiener_normals(M.seed[0], (uint64_t)k, (uint32_t)M.q);
    Normals4 b = a;
    if (WIDTH<V> == 2) b = wiener_normals(M.seed[1], (uint64_t)k, (uint32_t)M.q);
    w[0] = both<V>(a.a, b.a);
    w[1] = both<V>(a.b, b.b);
    w[2] = both<V>(a.c, b.c);
}

// The effective field at m; d: the dipolar field, formed here or given.
template <bool SPLIT, bool GIVEN, class V>
__device__ inline void field_at(const AdjArgs &A, AdjMember<V> &M, const V m[3], float s,
                                V h[3], V d[3])
{
    if (!GIVEN) {
        if (A.interactions) dip<SPLIT>(M, m, d);
        else d[0] = d[1] = d[2] = all<V>(0.f);
    }
    const V dot = mul2(dot3(m, M.ax), M.k);
    h[0] = fma2(dot, M.ax[0], d[0]);
    h[1] = fma2(dot, M.ax[1], d[1]);
    h[2] = fma2(all<V>(A.happ), all<V>(s), fma2(dot, M.ax[2], d[2]));
}

// one forward step (step index k, 1-based) of the float-float state hi + lo;
// d1, d2: the dipolar fields of its two stages
template <bool SPLIT, class V>
__device__ inline void fstep(const AdjArgs &A, AdjMember<V> &M, V hi[3], V lo[3],
                             int64_t k, V d1[3], V d2[3])
{
    V w[3];
    increments(M, k, w);
    const float2 s = A.stab ? __ldg(A.stab + (k - 1)) : make_float2(1.f, 1.f);
    const V ssr = mul2(all<V>(A.sq), M.srq), dt = all<V>(A.dt), al = all<V>(A.alpha);
    V h[3], v[3], f1[3], f2nd[3], xt[3];
    field_at<SPLIT, false>(A, M, hi, s.x, h, d1);
    for (int c = 0; c < 3; c++) v[c] = fma2(dt, h[c], mul2(ssr, w[c]));
    llg(f1, hi, al, v);
    for (int c = 0; c < 3; c++) xt[c] = add2(hi[c], f1[c]);
    field_at<SPLIT, false>(A, M, xt, s.y, h, d2);
    for (int c = 0; c < 3; c++) v[c] = fma2(dt, h[c], mul2(ssr, w[c]));
    llg(f2nd, xt, al, v);
    for (int c = 0; c < 3; c++)
        dd_add(hi[c], lo[c], fma2(all<V>(0.5f), f2nd[c], mul2(all<V>(0.5f), f1[c])));
}

template <class V>
__device__ inline void write_sample_a(const AdjArgs &A, const AdjMember<V> &M, int64_t s,
                                      const V hi[3], const V lo[3])
{
    if (!M.writes || !A.mx) return;
    const int64_t o = s * A.P + M.g;
    double *out[3] = {A.mx + o, A.my + o, A.mz + o};
    for (int c = 0; c < 3; c++) {
        out[c][0] = ((double)first(hi[c]) + (double)first(lo[c])) * A.out_scale[M.e];
        if (M.second)
            out[c][A.n] = ((double)last(hi[c]) + (double)last(lo[c])) * A.out_scale[M.e + 1];
    }
}

template <class V>
__device__ inline void write_ck(const AdjArgs &A, const AdjMember<V> &M, int64_t c,
                                const V hi[3], const V lo[3])
{
    if (!M.writes) return;
    V *o = (V *)A.ck + c * 6 * M.pairs + M.pair;
    for (int i = 0; i < 3; i++) {
        o[i * M.pairs] = hi[i];
        o[(3 + i) * M.pairs] = lo[i];
    }
}

// Moments m of step k (0-based) and, KEPT, the dipolar fields of its two stages
// into `seg`, the step's planes at `o`.
template <bool KEPT, class V>
__device__ inline void keep_fields(const AdjMember<V> &M, V *o, const V d1[3], const V d2[3])
{
    if (KEPT && M.writes)
        for (int i = 0; i < 3; i++) {
            o[(3 + i) * M.pairs] = d1[i];
            o[(6 + i) * M.pairs] = d2[i];
        }
}

template <class V>
__device__ inline void keep_moments(const AdjMember<V> &M, V *o, const V m[3])
{
    if (M.writes)
        for (int i = 0; i < 3; i++) o[i * M.pairs] = m[i];
}

// WHOLE: every step's moments and dipolar fields are kept for the sweep back,
// which then forms two sums a step, not the forward pass's two again as well (27
// particles, 2048 members, 512 steps: 5.4 -> 3.9 ms in all; 1000 members, 256
// steps: 2.30 -> 1.80).  The launch bounds leave registers for the loads that a
// sum's unrolled sources need in flight: left to itself the compiler took 64 to 87,
// and the pass was slower than the one without kept fields (us, 100 members: 60
// particles 994 -> 760, 128 4556 -> 2081; 27 particles 736 -> 629).
template <class V, int MAXT, bool SPLIT, bool WHOLE>
__global__ void __launch_bounds__(MAXT, MAXT == 128 ? 3 : 1) adj_forward_kernel(AdjArgs A)
{
    extern __shared__ float4 smem_a[];
    AdjMember<V> M;
    if (!setup_member<SPLIT>(A, M, smem_a)) return;
    const int64_t P = A.P;
    const int next = M.second ? A.n : 0;
    V hi[3], lo[3];
    for (int c = 0; c < 3; c++) {
        const double v0 = A.m0[c * P + M.g], v1 = A.m0[c * P + M.g + next];
        hi[c] = both<V>((float)v0, (float)v1);
        lo[c] = both<V>((float)(v0 - (double)first(hi[c])), (float)(v1 - (double)last(hi[c])));
    }
    if (!WHOLE) write_ck(A, M, 0, hi, lo);
    write_sample_a(A, M, 0, hi, lo);
    int64_t s_next = 1, ck = 0, next_ck = A.C;
    for (int64_t step = 1; step <= A.K; step++) {
        while (s_next < A.S && A.sched[s_next] == step) write_sample_a(A, M, s_next++, hi, lo);
        V d1[3], d2[3];
        V *o = WHOLE ? (V *)A.seg + (step - 1) * 9 * M.pairs + M.pair : nullptr;
        if (WHOLE) keep_moments(M, o, hi);
        fstep<SPLIT>(A, M, hi, lo, step, d1, d2);
        if (WHOLE) keep_fields<true>(M, o, d1, d2);
        if (!WHOLE && step == next_ck) {
            write_ck(A, M, ++ck, hi, lo);
            next_ck += A.C;
        }
    }
    bool bad[2] = {false, false};
    for (int c = 0; c < 3; c++) {
        bad[0] |= M.active && !isfinite(first(hi[c]));
        bad[1] |= M.active && !isfinite(last(hi[c]));
    }
    for (int i = 0; i < WIDTH<V>; i++) {
        const bool any = M.ms.cta ? (__syncthreads_or(bad[i]) != 0)
                                  : (__any_sync(M.ms.mask, bad[i]) != 0);
        if (M.q == 0 && M.half == 0 && A.status && (i == 0 || M.second))
            A.status[M.e + i] = any ? ST_NONFINITE : ST_OK;
    }
}

// reverse of step k (1-based) taken from the moments m = x_{k-1}.hi; KEPT: the
// dipolar fields d1, d2 of its stages are given
template <bool SPLIT, bool KEPT, class V>
__device__ inline void bstep(const AdjArgs &A, AdjMember<V> &M, const V m[3], int64_t k,
                             V lam[3], V G[5], V d1[3], V d2[3])
{
    V w[3];
    increments(M, k, w);
    const float2 s = A.stab ? __ldg(A.stab + (k - 1)) : make_float2(1.f, 1.f);
    const V ssr = mul2(all<V>(A.sq), M.srq), dt = all<V>(A.dt), al = all<V>(A.alpha);
    V h1[3], v1[3], f1[3], xt[3], h2[3], v2[3];
    field_at<SPLIT, KEPT>(A, M, m, s.x, h1, d1);
    for (int c = 0; c < 3; c++) v1[c] = fma2(dt, h1[c], mul2(ssr, w[c]));
    llg(f1, m, al, v1);
    for (int c = 0; c < 3; c++) xt[c] = add2(m[c], f1[c]);
    field_at<SPLIT, KEPT>(A, M, xt, s.y, h2, d2);
    for (int c = 0; c < 3; c++) v2[c] = fma2(dt, h2[c], mul2(ssr, w[c]));
    const V sw[3] = {mul2(M.srq, w[0]), mul2(M.srq, w[1]), mul2(M.srq, w[2])};
    const V inv_c = all<V>(A.c != 0.f ? 1.f / A.c : 0.f);
    const V inv_v = all<V>(1.f / first(M.vq));

    // stage 2
    V g2[3], mu2[3], lt[3] = {all<V>(0.f), all<V>(0.f), all<V>(0.f)}, eta2[3];
    for (int c = 0; c < 3; c++) g2[c] = mul2(all<V>(0.5f), lam[c]);
    MT(mu2, xt, al, g2);
    JmT_add(lt, xt, al, v2, g2);
    G[2] = add2(G[2], dFda(xt, v2, g2));
    for (int c = 0; c < 3; c++) eta2[c] = mul2(dt, mu2[c]);
    G[0] = add2(G[0], dot3(mu2, h2));
    G[1] = add2(G[1], dot3(mu2, sw));
    V de = mul2(M.k, dot3(M.ax, eta2));
    for (int c = 0; c < 3; c++) lt[c] = fma2(de, M.ax[c], lt[c]);
    if (A.interactions) {
        const V et[3] = {mul2(eta2[0], inv_v), mul2(eta2[1], inv_v), mul2(eta2[2], inv_v)};
        V dd[3];
        dip<SPLIT>(M, et, dd);
        for (int c = 0; c < 3; c++) lt[c] = fma2(M.vq, dd[c], lt[c]);
        G[4] = fma2(dot3(eta2, d2), inv_c, G[4]);
    }
    G[3] = fma2(eta2[2], all<V>(s.y), G[3]);

    // stage 1
    V g1[3], mu1[3], ln[3], eta1[3];
    for (int c = 0; c < 3; c++) {
        g1[c] = fma2(all<V>(0.5f), lam[c], lt[c]);
        ln[c] = add2(lam[c], lt[c]);
    }
    MT(mu1, m, al, g1);
    JmT_add(ln, m, al, v1, g1);
    G[2] = add2(G[2], dFda(m, v1, g1));
    for (int c = 0; c < 3; c++) eta1[c] = mul2(dt, mu1[c]);
    G[0] = add2(G[0], dot3(mu1, h1));
    G[1] = add2(G[1], dot3(mu1, sw));
    de = mul2(M.k, dot3(M.ax, eta1));
    for (int c = 0; c < 3; c++) ln[c] = fma2(de, M.ax[c], ln[c]);
    if (A.interactions) {
        const V et[3] = {mul2(eta1[0], inv_v), mul2(eta1[1], inv_v), mul2(eta1[2], inv_v)};
        V dd[3];
        dip<SPLIT>(M, et, dd);
        for (int c = 0; c < 3; c++) ln[c] = fma2(M.vq, dd[c], ln[c]);
        G[4] = fma2(dot3(eta1, d1), inv_c, G[4]);
    }
    G[3] = fma2(eta1[2], all<V>(s.x), G[3]);
    for (int c = 0; c < 3; c++) lam[c] = ln[c];
}

template <class V, int MAXT, bool SPLIT, bool KEPT>
__global__ void __launch_bounds__(MAXT, MAXT == 128 ? 3 : 1) adj_backward_kernel(AdjArgs A)
{
    extern __shared__ float4 smem_a[];
    AdjMember<V> M;
    if (!setup_member<SPLIT>(A, M, smem_a)) return;
    const int64_t N2 = M.pairs;
    V lam[3] = {all<V>(0.f), all<V>(0.f), all<V>(0.f)};
    double Gt[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    int64_t s_ptr = A.S - 1;
    const int64_t nseg = (A.K + A.C - 1) / A.C;
    for (int64_t c = nseg - 1; c >= 0; c--) {
        const int64_t k0 = c * A.C, k1 = (k0 + A.C < A.K) ? k0 + A.C : A.K;
        // per step the moments and, KEPT, the dipolar fields of its two stages:
        // the sweep back then forms two sums a step instead of four
        constexpr int PLANES = KEPT ? 9 : 3;
        V *sg = (V *)A.seg + M.pair;
        if (KEPT && A.whole) {
            sg += k0 * PLANES * N2;
        } else {
            V hi[3], lo[3];
            const V *ck = (const V *)A.ck + c * 6 * N2 + M.pair;
            for (int i = 0; i < 3; i++) {
                hi[i] = ck[i * N2];
                lo[i] = ck[(3 + i) * N2];
            }
            if (SPLIT) __syncthreads();  // the other warp has read the last segment
            for (int64_t k = k0; k < k1; k++) {
                V *o = sg + (k - k0) * PLANES * N2;
                keep_moments(M, o, hi);
                V d1[3], d2[3];
                fstep<SPLIT>(A, M, hi, lo, k + 1, d1, d2);
                keep_fields<KEPT>(M, o, d1, d2);
            }
            if (SPLIT) __syncthreads();
        }
        V G[5] = {all<V>(0.f), all<V>(0.f), all<V>(0.f), all<V>(0.f), all<V>(0.f)};
        for (int64_t k = k1 - 1; k >= k0; k--) {
            const V *in = sg + (k - k0) * PLANES * N2;
            V m[3], d1[3], d2[3];
            for (int i = 0; i < 3; i++) {
                m[i] = in[i * N2];
                if (KEPT) {
                    d1[i] = in[(3 + i) * N2];
                    d2[i] = in[(6 + i) * N2];
                }
            }
            bstep<SPLIT, KEPT>(A, M, m, k + 1, lam, G, d1, d2);
            // samples s >= 1 hold x_{sched[s]-1}: add their objective weights
            while (s_ptr >= 1 && A.sched[s_ptr] - 1 > k) s_ptr--;
            while (s_ptr >= 1 && A.sched[s_ptr] - 1 == k) {
                const float wz = (float)A.wz[s_ptr--];
                lam[2] = add2(lam[2], all<V>(wz));
            }
        }
        for (int i = 0; i < 5; i++) Gt[i] += (double)first(G[i]) + (M.second ? (double)last(G[i]) : 0.0);
    }
    if (M.writes)
        for (int i = 0; i < 5; i++) atomicAdd(&A.grad[i], Gt[i]);
}

}  // namespace

namespace adj {


struct Launch {
    dim3 grid, block;
    size_t shmem;
    bool two, split;  // two members per thread; two warps per sum
};

static Launch shape(int n, int64_t E, bool interactions)
{
    Launch L;
    const int mpw = n <= 32 ? 32 / n : 1, wpm = n <= 32 ? 1 : (n + 31) / 32;
    const int64_t warps1 = (E + mpw - 1) / mpw * wpm;  // with one member per thread
    // Two members per thread halve the instructions and table reads of a sum
    // and lengthen a warp's chain: the better form once the warps (of the other
    // form) about fill the sub-partitions and the sums are most of the work.
    // With few warps the chain is what counts, and two warps share the sources
    // (the rest of a step both do).  Forward and backward, 256 steps, ms with
    // one member / two members / two warps: 27 particles, 2048 members 3.93 /
    // 2.23 / 4.56; 1000 1.58 / 1.61 / 2.50; 100 1.11 / 1.41 / 1.05; 13, 2500
    // 1.63 / 1.68 / 2.83; 13, 1000 1.16 / 1.32 / 1.21; 8, 8000 3.78 / 2.77 / 4.49;
    // 8, 1000 1.08 / 1.26 / 0.90; 60, 500 2.70 / 2.55; 60, 200 1.96 / 2.39.
    L.two = warps1 >= 1000 && warps1 * n >= 16000;
    L.split = !L.two && n <= 32 && interactions && n >= 5 && warps1 <= 400;
    const int W = L.two ? 2 : 1;
    const int64_t items = (E + W - 1) / W;
    int64_t slots = 1;
    if (n > 32) {
        L.block = dim3(32 * wpm);
        L.grid = dim3((unsigned)items);
    } else {
        // one warp per CTA while every warp has a sub-partition or a few share one
        const int warps = (items + mpw - 1) / mpw <= 4 * sub_partitions() ? 1 : 4;
        L.block = dim3(L.split ? 64 : 32 * warps);
        const int64_t per_block = (int64_t)(L.split ? 1 : warps) * mpw;
        L.grid = dim3((unsigned)((items + per_block - 1) / per_block));
        slots = (L.split ? 2 : 1) * per_block;
    }
    L.shmem = (slots * n + (slots * n + 1) / 2) * sizeof(float4) +
              (L.split ? 2 * 192 * W * sizeof(float) : 0);
    return L;
}

template <class V>
static void run(const Launch &L, const AdjArgs &A, bool backward, bool kept, cudaStream_t stream)
{
    const bool small = L.block.x <= 128;  // small CTAs may use more registers
    auto go = [&](auto kernel) { kernel<<<L.grid, L.block, L.shmem, stream>>>(A); };
    if constexpr (WIDTH<V> == 1)
        if (L.split) {
            if (!backward && A.whole) go(adj_forward_kernel<V, 64, true, true>);
            else if (!backward) go(adj_forward_kernel<V, 64, true, false>);
            else if (kept) go(adj_backward_kernel<V, 64, true, true>);
            else go(adj_backward_kernel<V, 64, true, false>);
            return;
        }
    if (!backward && A.whole) {
        if (small) go(adj_forward_kernel<V, 128, false, true>);
        else go(adj_forward_kernel<V, 512, false, true>);
    } else if (!backward) {
        if (small) go(adj_forward_kernel<V, 128, false, false>);
        else go(adj_forward_kernel<V, 512, false, false>);
    } else if (kept) {
        if (small) go(adj_backward_kernel<V, 128, false, true>);
        else go(adj_backward_kernel<V, 512, false, true>);
    } else {
        if (small) go(adj_backward_kernel<V, 128, false, false>);
        else go(adj_backward_kernel<V, 512, false, false>);
    }
}

}  // namespace adj

cudaError_t launch_adjoint(const AdjointArgs &a, bool backward, cudaStream_t stream)
{
    AdjArgs A;
    A.E = a.p.E; A.P = a.p.P; A.S = a.p.S; A.K = a.K;
    A.n = a.p.n; A.C = a.C; A.interactions = a.interactions;
    A.members = a.p.members; A.m0 = a.p.m0; A.axes = a.p.axes; A.k_red = a.p.k_red;
    A.sr = a.p.sr; A.v_red = a.v_red; A.pr = a.p.pr; A.stab = (const float2 *)a.stab;
    A.happ = a.happ; A.dt = a.dt; A.sq = a.sq; A.alpha = a.alpha; A.c = a.c;
    A.sched = a.p.sched; A.ck = a.ck; A.seg = a.seg; A.whole = a.whole; A.out_scale = a.p.out_scale;
    A.mx = a.p.mx; A.my = a.p.my; A.mz = a.p.mz; A.wz = a.wz; A.grad = a.grad;
    A.status = a.p.status;
    if (A.E == 0) return cudaSuccess;
    const adj::Launch L = adj::shape(A.n, A.E, A.interactions != 0);
    if (L.two) adj::run<float2>(L, A, backward, a.kept, stream);
    else adj::run<float>(L, A, backward, a.kept, stream);
    return cudaGetLastError();
}

}  // namespace magpy
