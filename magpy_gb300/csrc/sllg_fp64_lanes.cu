// sllg_fp64_lanes.cu -- the FP64-faithful sLLG kernel for small ensembles:
// several lanes per particle (compiled with -fmad=false).
//
// What bounds a small ensemble: an FP64 instruction takes 64 issue cycles of a
// warp's sub-partition however many of its lanes are active, and one warp
// fills that pipe.  With one thread per particle (sllg_fp64.cu) a Heun step is
// about 220 FP64 instructions and an implicit step 335 a Newton iteration,
// while most of the chip idles.  The LLG expressions are cyclic in the three
// components, so here the lanes of a group compute one component (row) each:
// about 75 FP64 instructions a Heun step, 155 (4 lanes) or 120 (16) a Newton
// iteration.  2000 Heun steps of 1000 single particles: 17.0 -> 6.9 ms; 250
// implicit steps of one particle: 66.9 -> 30.1 ms.  Every product and sum keeps the
// association of the reference's expressions (lib/llg.cpp, lib/field.cpp,
// lib/integrators.cpp), which are not all cyclic: where the order of a sum or
// a product follows the absolute component, a lane selects its operands by its
// component.  The trajectories have the same bits as sllg_fp64.cu's.
//
// COLS = 1: 4 lanes per particle (component c = 0, 1, 2; the fourth repeats
// c = 2), 8 particles per warp.  COLS = 3 (implicit, one or two particles per
// member): 16 lanes per particle, lane 4 k + c computing entry (c, k) of the
// Newton matrix, the rest as COLS = 1.
#include <algorithm>
#include "common.cuh"
#include "fp64_common.cuh"
#include "llg64.cuh"
#include "plan.hpp"

namespace magpy {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// A lane's place: component c, the next two v = c + 1, w = c + 2 (mod 3), the
// first lane of its particle's group, and its row-column entry.
struct Lane {
    int c, v, w, base, col;
    int vs;          // particle slot whose state the lane holds
    bool is0, is1, is2;
    __device__ inline double of(double x, int comp) const { return __shfl_sync(FULL, x, base + comp); }
    __device__ inline double next(double x) const { return of(x, v); }
    __device__ inline double prev(double x) const { return of(x, w); }
};

// x, y, z in a lane's cyclic order (own component, next, previous) -> the
// order of the absolute component.
__device__ inline void absolute(const Lane &L, double x, double y, double z, double o[3])
{
    o[0] = L.is0 ? x : L.is1 ? z : y;
    o[1] = L.is0 ? y : L.is1 ? x : z;
    o[2] = L.is0 ? z : L.is1 ? y : x;
}

struct ParticleL {
    double ax, k, sr, alpha, asr;
    // field-Jacobian entries of row v, w, c: column c, v, w (COLS = 1) or the
    // lane's own column in element 0
    double jv[3], jw[3], jc[3];
};

struct MemberL {
    const MemberDev *d;
    const double *pt, *rt;
    double *sm;      // [slots][3] moments of the warp
    int n, q, first; // particle of the member, first slot of the member
    bool inter, writes;
};

// eff_field of sllg_fp64.cu, component c.
__device__ inline double field_of(const Lane &L, const MemberL &M, const ParticleL &pa, double s,
                                  double hz)
{
    const double p = s * pa.ax;
    double dot = L.of(p, 0) + L.of(p, 1) + L.of(p, 2);
    dot *= pa.k;
    double h = plus_zero(dot * pa.ax);
    h = h + (L.is2 ? hz : -0.0);  // adding -0 changes nothing
    if (M.inter) {
        if (M.writes) M.sm[3 * L.vs + L.c] = s;
        __syncwarp();
        const int n = M.n, q = M.q;
        for (int j = 0; j < n; j++) {
            const double mj = M.sm[3 * (M.first + j) + L.c];
            const double P = __ldg(M.pt + (size_t)j * n + q);
            const double r = __ldg(M.rt + ((size_t)L.c * n + j) * n + q);
            const double pr = mj * r;
            const double d = L.of(pr, 0) + L.of(pr, 1) + L.of(pr, 2);
            const double t = h + P * (3 * d * r - mj);
            h = j == q ? h : t;
        }
        __syncwarp();
    }
    return h;
}

// llg::drift and llg::diffusion, row c: a, and B's entries in the lane's
// cyclic order (columns c, v, w).
struct Stage {
    double mv, mw, hv, hw;  // moments and field of the other components
    double s, q, X, Y;      // m_v^2 + m_w^2, m_v h_v + m_w h_w, m_w h_v, m_v h_w
    double a, bd, bn, bp;
};

__device__ inline Stage stage_of(const Lane &L, const ParticleL &pa, double m, double h)
{
    Stage S;
    S.mv = L.next(m);
    S.mw = L.prev(m);
    S.hv = L.next(h);
    S.hw = L.prev(h);
    const double sq = m * m, mh = m * h;
    S.s = L.next(sq) + L.prev(sq);
    S.q = L.next(mh) + L.prev(mh);
    S.X = S.mw * S.hv;
    S.Y = S.mv * S.hw;
    S.a = (S.X - S.Y) + pa.alpha * (h * S.s - m * S.q);
    // alpha m_i m_j, i < j, of the pair {c, v}; {w, c} is the previous lane's
    const double A = pa.alpha * (L.is2 ? S.mv : m) * (L.is2 ? m : S.mv);
    const double Aw = L.prev(A);
    S.bd = pa.asr * S.s;
    S.bn = pa.sr * (S.mw - A);
    S.bp = -(pa.sr * (S.mv + Aw));
    return S;
}

// integrator::heun, lib/integrators.cpp:372-405, component c.
__device__ inline double heun_lane(const Lane &L, const MemberL &M, const ParticleL &pa, double px,
                                   double w, double hz1, double hz2)
{
    const double dt = M.d->dt, sq = M.d->sqrt_dt;
    const double wv = L.next(w), ww = L.prev(w);
    double o[3];
    const Stage A = stage_of(L, pa, px, field_of(L, M, pa, px, hz1));
    absolute(L, A.bd * w * sq, A.bn * wv * sq, A.bp * ww * sq, o);
    double xt = px + dt * A.a;
    xt += o[0];
    xt += o[1];
    xt += o[2];
    const Stage B = stage_of(L, pa, xt, field_of(L, M, pa, xt, hz2));
    const double kw = 0.5 * w * sq;
    absolute(L, kw * (B.bd + A.bd), L.next(kw) * (B.bn + A.bn), L.prev(kw) * (B.bp + A.bp), o);
    double x = px + 0.5 * dt * (B.a + A.a);
    x += o[0];
    x += o[1];
    x += o[2];
    return x;
}

// member_sumsq of sllg_fp64.cu: per particle the components in order, then the
// pairwise tree over the member's particles.
__device__ inline double sumsq_lane(const Lane &L, const MemberL &M, int lanes, int p2, double x)
{
    const double sq = x * x;
    double s = L.of(sq, 0) + L.of(sq, 1) + L.of(sq, 2);
    if (M.n == 1) return s;
    for (int stride = p2 >> 1; stride >= 1; stride >>= 1) {
        const bool add = M.q < stride && M.q + stride < M.n;
        const double t = __shfl_sync(FULL, s, lanes * (L.vs + (add ? stride : 0)));
        if (add) s = s + t;
    }
    return __shfl_sync(FULL, s, lanes * M.first);
}

// Entry (c, column o of the cyclic order) of the Newton matrix I - 0.5 a' -
// 0.5 sum_k b'_k dwm_k (implicit_step of sllg_fp64.cu): hc, hv, hw = dwm / 2.
__device__ inline double newton_entry(const Lane &L, const ParticleL &pa, const Stage &S, double m,
                                      double gv, double gw, double jv, double jw, double jc, int o,
                                      double cu, double cv, double cw, const double hd[3])
{
    const bool d = o == 0, n = o == 1;
    // llg::drift_jacobian: sums run over the rows v, w in absolute order, which
    // for c = 1 is w, v; a diagonal entry has no first term (-0 adds nothing)
    const double X1 = S.mw * jv, Y1 = -(S.mv * jw), X2 = S.mv * jv, Y2 = S.mw * jw;
    const double base = d ? -0.0 : n ? -S.hw : S.hv;
    const double hb = d ? -0.0 : n ? S.hv : S.hw;
    const double G = d ? S.q : n ? gv : gw;
    const double out = (base + (L.is1 ? Y1 : X1)) + (L.is1 ? X1 : Y1);
    const double in = (hb + (L.is1 ? Y2 : X2)) + (L.is1 ? X2 : Y2);
    const double D = out + pa.alpha * (fma(d ? -1.0 : 2.0, G, S.s * jc) - m * in);
    double J = fma(-0.5, D, d ? 1.0 : 0.0);
    // llg::diffusion_jacobian with its entries [4] and [25]; A: k = c, B: k = v,
    // C: k = w; a term that is not there has the factor 0
    const double A = (n ? cv : L.is2 ? cu : cw) * hd[0];
    const double B = (d ? cv : n ? (L.is0 ? cw : cu) : pa.sr) * hd[1];
    const double C = (d ? cw : n ? pa.sr : cu) * hd[2];
    const double fA = d ? 0.0 : -2.0, fB = o == 2 ? -1.0 : 1.0;
    double t[3], f[3];
    absolute(L, A, B, C, t);
    absolute(L, fA, fB, 1.0, f);
    J = fma(f[0], t[0], J);
    J = fma(f[1], t[1], J);
    return fma(f[2], t[2], J);
}

// f64::solve3_bits with row c of the matrix and right-hand side in lane c;
// the result's component c.  Returns 0 or non-zero for a zero pivot, the same
// in every lane of the particle.
__device__ inline int solve_lanes(const Lane &L, double A0, double A1, double A2, double B,
                                  double &sol)
{
    using f64::is_zero;
    using f64::larger_mag;
    int info = 0;
    const double g0 = L.of(A0, 0), g1 = L.of(A0, 1), g2 = L.of(A0, 2);
    const bool p1 = larger_mag(g1, g0);
    const bool p2 = larger_mag(g2, p1 ? g1 : g0);
    const int r0 = p2 ? 2 : p1 ? 1 : 0;
    // the rows at positions 1 and 2 after the swap with row 0
    int ra = (p1 && !p2) ? 0 : 1, rb = p2 ? 0 : 2;
    const double P0 = p2 ? g2 : p1 ? g1 : g0;
    const double P1 = L.of(A1, r0), P2 = L.of(A2, r0), PB = L.of(B, r0);
    if (is_zero(P0)) info = 1;
    const bool below = L.c != r0;
    const double l = (below && !info ? A0 : 1.0) / (info ? 1.0 : P0);
    const double A1s = A1 - l * P1, A2s = A2 - l * P2, Bs = B - PB * l;
    A1 = below ? A1s : A1;
    A2 = below ? A2s : A2;
    B = below ? Bs : B;
    const double ga = L.of(A1, ra), gb = L.of(A1, rb);
    const bool p = larger_mag(gb, ga);
    const int r1 = p ? rb : ra, r2 = p ? ra : rb;
    const double Q1 = p ? gb : ga;
    const double Q2 = L.of(A2, r1), QB = L.of(B, r1);
    if (!info && is_zero(Q1)) info = 2;
    const bool last = L.c == r2;
    const double l2 = (last && !info ? A1 : 1.0) / (info ? 1.0 : Q1);
    const double A2t = A2 - l2 * Q2, Bt = B - QB * l2;
    A2 = last ? A2t : A2;
    B = last ? Bt : B;
    const double Z = L.of(A2, r2), ZB = L.of(B, r2);
    if (!info && is_zero(Z)) info = 3;
    const double x2 = (info ? 0.0 : ZB) / (info ? 1.0 : Z);
    B = B - x2 * A2;
    const double x1 = (info ? 0.0 : L.of(B, r1)) / (info ? 1.0 : Q1);
    B = B - x1 * P1;
    const double x0 = (info ? 0.0 : L.of(B, r0)) / (info ? 1.0 : P0);
    sol = L.is0 ? x0 : L.is1 ? x1 : x2;
    return info;
}

// integrator::implicit_midpoint, component c (implicit_step of sllg_fp64.cu).
// The warp's members iterate together; one that has stopped keeps its state.
template <int COLS>
__device__ inline int32_t implicit_lane(const Lane &L, const MemberL &M, const ParticleL &pa,
                                        int p2, double &x, double px, double w, double hz1,
                                        double hz2)
{
    constexpr int LANES = COLS == 1 ? 4 : 16;
    const double dt = M.d->dt, sq = M.d->sqrt_dt, Ah = M.d->Ah;
    const double lo = (w < Ah) ? w : Ah;
    const double dwm = ((-Ah < lo) ? lo : -Ah) * sq;
    const double hw = 0.5 * dwm;
    double o[3];
    {
        const Stage S = stage_of(L, pa, px, field_of(L, M, pa, px, hz1));
        absolute(L, S.bd * dwm, S.bn * L.next(dwm), S.bp * L.prev(dwm), o);
        double g = S.a * dt;
        g += o[0];
        g += o[1];
        g += o[2];
        x = (g + px) / 2;
    }
    const double tol = M.d->eps * sqrt(sumsq_lane(L, M, LANES, p2, x)), tol2 = tol * tol;
    bool going = 2 * tol > tol;
    int64_t iter = M.d->max_iter;
    int32_t flag = ST_OK;
    const double hdt = 0.5 * dt;
    const double hd[3] = {hw, L.next(hw), L.prev(hw)};
    // while (going && (iter-- > 0)), per member
    for (;;) {
        if (going) going = iter-- > 0;
        if (!__any_sync(FULL, going)) break;
        const double m = x;
        const Stage S = stage_of(L, pa, m, field_of(L, M, pa, m, hz2));
        absolute(L, S.bd * hd[0], S.bn * hd[1], S.bp * hd[2], o);
        double F = (m - S.a * hdt) - px;
        F -= o[0];
        F -= o[1];
        F -= o[2];
        const double gv = L.prev(S.X), gw = L.next(S.Y);  // m_v h_c, m_w h_c
        const double cu = pa.asr * m, cv = L.next(cu), cw = L.prev(cu);
        double J[3];
        if (COLS == 1) {
            double e[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                e[k] = newton_entry(L, pa, S, m, gv, gw, pa.jv[k], pa.jw[k], pa.jc[k], k, cu, cv,
                                    cw, hd);
            absolute(L, e[0], e[1], e[2], J);
        } else {
            const int k = L.col - L.c;
            const double e = newton_entry(L, pa, S, m, gv, gw, pa.jv[0], pa.jw[0], pa.jc[0],
                                          k < 0 ? k + 3 : k, cu, cv, cw, hd);
            for (int c = 0; c < 3; c++) J[c] = L.of(e, 4 * c + L.c);
        }
        double sol;
        const int info = solve_lanes(L, J[0], J[1], J[2], -F, sol);
        // any particle of the member
        bool sing = false;
        for (int k = 0; k < M.n; k++)
            sing |= __shfl_sync(FULL, info, LANES * (M.first + k)) != 0;
        const double err2 = sumsq_lane(L, M, LANES, p2, sol);
        if (going) {
            if (sing) {
                flag = ST_SINGULAR;
                x = -F;
                going = false;
            } else {
                x = sol + m;
                going = norm_above(err2, tol, tol2);
            }
        }
    }
    if (flag == ST_OK && iter == -1) flag = ST_NEWTON_MAXITER;
    x = 2 * x - px;
    return flag;
}

template <bool IMPLICIT, int COLS>
__global__ void __launch_bounds__(32) sllg_fp64_lanes_kernel(DevPlan p)
{
    constexpr int LANES = COLS == 1 ? 4 : 16, SLOTS = 32 / LANES;
    __shared__ double sm[3 * SLOTS];
    const int n = p.n, lane = threadIdx.x, mpw = p.members_per_warp;
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    const int64_t e0 = (int64_t)blockIdx.x * mpw;
    const int members = (int)(p.E - e0 < mpw ? p.E - e0 : mpw);
    // lanes without a particle of their own repeat another's (and write nothing)
    const int slot = lane / LANES, used = members * n;
    Lane L;
    L.vs = slot % used;
    const int in = lane % 4;
    L.c = in == 3 ? 2 : in;
    L.v = L.c == 2 ? 0 : L.c + 1;
    L.w = L.c == 0 ? 2 : L.c - 1;
    L.is0 = L.c == 0;
    L.is1 = L.c == 1;
    L.is2 = L.c == 2;
    L.base = L.vs * LANES;
    L.col = COLS == 1 ? 0 : min((lane % LANES) >> 2, 2);
    MemberL M;
    M.n = n;
    M.q = L.vs % n;
    M.first = L.vs - M.q;
    const int64_t e = e0 + L.vs / n;
    const MemberDev *md = p.members + e;
    M.d = md;
    M.pt = p.pt + md->cluster_off;
    M.rt = p.rt + 3 * md->cluster_off;
    M.sm = sm;
    M.inter = md->interactions && n > 1;
    M.writes = slot < used && lane % LANES < 3;
    const int64_t P = p.P, g = md->pbase + M.q;
    ParticleL pa;
    pa.ax = p.axes[L.c * P + g];
    pa.k = p.k_red[g];
    pa.sr = p.sr[g];
    pa.alpha = md->alpha;
    pa.asr = pa.alpha * pa.sr;
    if (IMPLICIT) {
        const int col[3] = {L.c, L.v, L.w};
        for (int k = 0; k < 3; k++) {
            const int j = COLS == 1 ? col[k] : L.col;
            pa.jv[k] = p.hj[(3 * L.v + j) * P + g];
            pa.jw[k] = p.hj[(3 * L.w + j) * P + g];
            pa.jc[k] = p.hj[(3 * L.c + j) * P + g];
        }
    }
    double x = p.m0[L.c * P + g], px = x;
    const double scale = p.out_scale[e];
    double *out = p.mx ? (L.is0 ? p.mx : L.is1 ? p.my : p.mz) + g : nullptr;
    if (!M.writes) out = nullptr;
    const int64_t S = p.S;
    const int64_t *sched = p.sched + md->sched_off;
    const double *noise = p.noise ? p.noise + md->noise_off : nullptr;
    const int64_t per_step = 3 * (int64_t)n;
    AppliedField af;
    {
        const MemberDev *d0 = p.members + e0;
        af.init(*md, __all_sync(FULL, md->dt == d0->dt && md->happ == d0->happ &&
                                          md->fapp == d0->fapp && md->shape == d0->shape));
    }
    if (out) out[0] = x * scale;  // sample 0, simulation.cpp:212-219
    int32_t status = ST_OK;
    uint64_t step = 0;
    int64_t s = 1;
    // every member of the launch takes the same steps and samples
    for (; s < S; s++) {
        const int64_t ks = sched[s];
        while ((int64_t)step < ks) {
            px = x;
            step++;
            double w;
            if (noise) {
                if ((int64_t)step * per_step > md->noise_len) {
                    status |= ST_NOISE_EXHAUSTED;
                    step--;
                    goto finished;
                }
                w = noise[(int64_t)(step - 1) * per_step + 3 * M.q + L.c];
            } else {
                const Normals4 r = wiener_normals(md->seed, step, (uint32_t)M.q);
                w = L.is0 ? r.a : L.is1 ? r.b : r.c;
            }
            double hz1, hz2;
            af.at<IMPLICIT>(*md, (int64_t)step, hz1, hz2);
            if (IMPLICIT)
                status |= implicit_lane<COLS>(L, M, pa, p2, x, px, w, hz1, hz2);
            else
                x = heun_lane(L, M, pa, px, w, hz1, hz2);
            if (md->renorm) {  // simulation.cpp:379-387
                const double sq = x * x;
                x = x / sqrt(L.of(sq, 0) + L.of(sq, 1) + L.of(sq, 2));
            }
        }
        if (out) out[s * P] = px * scale;  // zero-order hold, simulation.cpp:398-405
    }
finished:
    if (out)  // samples a stopped member never reached
        for (; s < S; s++) out[s * P] = NAN;
    const unsigned bad = __ballot_sync(FULL, !isfinite(x));
    for (int k = 0; k < n; k++)
        if ((bad >> (LANES * (M.first + k))) & 7u) status |= ST_NONFINITE;
    if (slot < used && lane % LANES == 0 && M.q == 0) {
        if (p.status) p.status[e] = status;
        if (p.steps) p.steps[e] = (int64_t)step;
    }
}

}  // namespace

// The launcher's choice (no launch shape set): a warp instruction costs the
// same for 8 particles as for 32, so several lanes per particle pay while the
// ensemble's warps find sub-partitions of their own -- with 75 instructions a
// Heun step instead of 220, up to two warps each.
static int lanes_cols(const DevPlan &p)
{
    if (p.block_warps > 0 || p.members_per_warp > 0 || !p.one_schedule || p.n > 8) return 0;
    const int64_t warps = (p.E + 8 / p.n - 1) / (8 / p.n), subs = sub_partitions();
    if (p.use_implicit && p.n <= 2 && (p.E + 2 / p.n - 1) / (2 / p.n) <= subs) return 3;
    return warps <= (p.use_implicit ? subs : 2 * subs) ? 1 : 0;
}

bool fp64_lanes_fit(const DevPlan &p) { return lanes_cols(p) > 0; }

cudaError_t launch_fp64_lanes(const DevPlan &p, cudaStream_t stream)
{
    const int cols = lanes_cols(p);
    DevPlan q = p;
    // members apart where every warp still has a sub-partition
    const int64_t most = (cols == 1 ? 8 : 2) / p.n, subs = sub_partitions();
    q.members_per_warp = (int)std::min<int64_t>(most, std::max<int64_t>(1, (p.E + subs - 1) / subs));
    const unsigned grid = (unsigned)((p.E + q.members_per_warp - 1) / q.members_per_warp);
    if (!p.use_implicit) sllg_fp64_lanes_kernel<false, 1><<<grid, 32, 0, stream>>>(q);
    else if (cols == 1) sllg_fp64_lanes_kernel<true, 1><<<grid, 32, 0, stream>>>(q);
    else sllg_fp64_lanes_kernel<true, 3><<<grid, 32, 0, stream>>>(q);
    return cudaGetLastError();
}

}  // namespace magpy
