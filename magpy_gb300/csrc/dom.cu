// dom.cu -- two-state master equation ("discrete orientation model") for a
// batch of independent particles, one thread per particle or five.
//
// Path restated: magpy/core.pyx:205-278 simulate_dom ->
// simulation::dom_ensemble_dynamics (lib/simulation.cpp:659-767) ->
// integrator::rk45 (lib/integrators.cpp:152-251) -> dom::master_equation_with_update
// (lib/dom.cpp:79-97) -> dom::transition_matrix (lib/dom.cpp:33-59) and the
// 2x2 product of stochastic::master_equation (lib/stochastic_processes.cpp:18-25).
//
// FP64 throughout, compiled without FMA contraction, in the reference's
// operation order; per-particle constants of the transition matrix (sigma,
// tau_N, its sqrt(pi)/sigma^1.5 factor) are computed once per particle, which
// yields the same values as recomputing them inside every evaluation.  The
// device's exp/pow/sin differ from the host libm by a few ulp, so results
// agree with the reference to rounding, not bit for bit.
//
// The reference's retry loop and sampling loop have no bound; here each step
// gives up after MAX_ATTEMPTS rejected trials and each particle after
// max_steps steps, with a status bit, so a NaN never turns into a spin.
#include <cmath>
#include "common.cuh"
#include "plan.hpp"
#include "rules.hpp"

namespace magpy {

namespace {

constexpr double KB_D = 1.38064852e-23;  // include/constants.hpp:10-12
constexpr double GYRO_D = 1.76086e11;
// One warp per CTA (DOM_THREADS, rules.hpp): the step counts of particles differ by
// orders of magnitude, so the launch (heaviest warps first) leaves the balancing of
// the SMs' FP64 pipes to the CTA scheduler.

struct DomParams {
    double hpre;   // (tau_N sqrt(pi)) / sigma^1.5
    double sigma;  // K V / kB / T
    double h, f;   // reduced field amplitude, frequency (Hz)
};

__device__ inline double dom_field(int shape, double t, double h, double f, int64_t ncomp)
{
    switch (shape) {
    case 2: return h;                                          // field.cpp:23-26
    case 0: return h * sin(2 * M_PI * f * t);                  // field.cpp:37-40
    case 1: return h * (int(t * f * 2) % 2 ? -1 : 1);          // field.cpp:51-54
    case 3: {                                                  // field.cpp:67-79
        double field = 0;
        for (unsigned int k = 1; k < (unsigned int)ncomp + 1; k++)
            field += sin(2 * M_PI * (2 * k - 1) * f * t) / (2 * k - 1);
        field *= 4 / M_PI * h;
        return field;
    }
    default: return NAN;
    }
}

// The rates of W(h(t)) = [[-r2, r1], [r2, -r1]]: lib/dom.cpp:33-59.
struct Rates { double r1, r2; };
__device__ inline Rates dom_rates(double t, const DomParams &q, int shape, int64_t ncomp)
{
    const double h = dom_field(shape, t, q.h, q.f, ncomp);
    const double e1 = q.sigma * (1 - h) * (1 - h);
    const double e2 = q.sigma * (1 + h) * (1 + h);
    const double pref = q.hpre / (1 - h * h);
    const double inv = 1.0 / pref;
    return Rates{inv * (1 - h) * exp(-e1), inv * (1 + h) * exp(-e2)};
}

// dp/dt = W p, component 0 (lib/dom.cpp:79-97; the row-major 2x2 product as
// the project's dgemv shim sums it).  Component 1 is its negative: the same
// two products, subtracted the other way round.
__device__ inline double dom_deriv(const Rates &w, double x0, double x1)
{
    return w.r1 * x1 - w.r2 * x0;
}

// One trial of the Cash-Karp RK45 step (lib/integrators.cpp:152-251;
// coefficients: J. R. Cash, A. H. Karp, ACM TOMS 16 (1990) 201-222) from `cur`
// with step h: the next state and the scaled error.  rate(s): the rates at
// stage s.  The stages' increments of the two components are each other's
// negative, so they are formed once.
template <class Rate>
__device__ inline double dom_trial(double next[2], double h, const double cur[2], double tol,
                                   const Rate &rate)
{
    const double c11 = 0.2, c21 = 3.0 / 40.0, c22 = 9.0 / 40.0, c31 = 3.0 / 10.0,
                 c32 = -9.0 / 10.0, c33 = 6.0 / 5.0, c41 = -11.0 / 54.0, c42 = 2.5,
                 c43 = -70.0 / 27.0, c44 = 35.0 / 27.0, c51 = 1631.0 / 55296.0,
                 c52 = 175.0 / 512.0, c53 = 575.0 / 13824.0, c54 = 44275.0 / 110592.0,
                 c55 = 253.0 / 4096.0;
    const double x11 = 37.0 / 378.0, x13 = 250.0 / 621.0, x14 = 125.0 / 594.0,
                 x16 = 512.0 / 1771.0;
    const double x21 = 2825.0 / 27648.0, x23 = 18575.0 / 48384.0, x24 = 13525.0 / 55296.0,
                 x25 = 277.0 / 14336.0, x26 = 0.25;
    double d;
    const double k1 = dom_deriv(rate(0), cur[0], cur[1]);
    d = k1 * h * c11;
    const double k2 = dom_deriv(rate(1), cur[0] + d, cur[1] - d);
    d = h * (c21 * k1 + c22 * k2);
    const double k3 = dom_deriv(rate(2), cur[0] + d, cur[1] - d);
    d = h * (c31 * k1 + c32 * k2 + c33 * k3);
    const double k4 = dom_deriv(rate(3), cur[0] + d, cur[1] - d);
    d = h * (c41 * k1 + c42 * k2 + c43 * k3 + c44 * k4);
    const double k5 = dom_deriv(rate(4), cur[0] + d, cur[1] - d);
    d = h * (c51 * k1 + c52 * k2 + c53 * k3 + c54 * k4 + c55 * k5);
    const double k6 = dom_deriv(rate(5), cur[0] + d, cur[1] - d);
    d = h * (x11 * k1 + x13 * k3 + x14 * k4 + x16 * k6);
    const double tmp[2] = {cur[0] + d, cur[1] - d};
    d = h * (x21 * k1 + x23 * k3 + x24 * k4 + x25 * k5 + x26 * k6);
    next[0] = cur[0] + d;
    next[1] = cur[1] - d;
    // std::pow(x, 2) compiles to x * x in the reference build (exact), and
    // std::pow(x, 0.5) of a non-negative finite x is within half an ulp of
    // the correctly rounded sqrt, which the device computes exactly
    const double mag = sqrt(cur[0] * cur[0] + cur[1] * cur[1]);
    const double e0 = tmp[0] - next[0], e1 = tmp[1] - next[1];
    return sqrt(e0 * e0 + e1 * e1) / (2.0 * tol * (1 + mag));
}

// The step after an accepted one of scaled error err < 1: min(5, 0.84
// err^-0.2) h, at most max_dt.  The power (about as long as four exponentials)
// is left out where it cannot matter: below 1.3e-4 it gives more than 5, and
// from a step at the limit an error below 0.84^5 = 0.418 leads past the limit.
__device__ inline double dom_next_step(double h, double err, double max_dt)
{
    // err is not negative: its high word orders like its value
    const int eh = __double2hiint(err);
    double hf;
    if (eh < 0x3f210000) {  // 1.297e-4
        hf = 5.0;
    } else if (__double_as_longlong(h) == __double_as_longlong(max_dt) && eh < 0x3fda0000) {
        return max_dt;  // 0.406
    } else {
        hf = 0.84 * pow(err, -0.2);
        hf = hf > 5 ? 5.0 : hf;
    }
    return hf * h;
}

__device__ inline double dom_shorter_step(double h, double err)
{
    double hf = 0.84 * pow(err, -0.2);
    hf = fabs(hf) < 0.1 ? 0.1 : hf;
    return h * hf;
}

// Stages 1..5 are at t + h * stage_time (lib/integrators.cpp:152-251).  Stage 4's is the time of the
// next step, so the rates found there are that step's first; a rejected step's
// first ones stay.
__device__ inline double stage_time(int s)
{
    return s == 1 ? 0.2 : s == 2 ? 0.3 : s == 3 ? 0.6 : s == 4 ? 1.0 : 7.0 / 8.0;
}

// One particle's state and outputs.
struct DomRun {
    DomParams q;
    double hk, t, t_last, dt, last[2], next[2];
    int64_t step, sample, e;
    int32_t status;
};

__device__ inline void dom_begin(DomRun &R, const DomArgs &a, int64_t e, bool write)
{
    const DomMember m = a.members[e];
    const double sigma = m.k * m.v / KB_D / m.T;
    const double taun = m.v * m.ms * (1 + m.alpha * m.alpha) / 2.0 / GYRO_D / m.alpha / KB_D / m.T;
    R.q = DomParams{taun * sqrt(M_PI) / pow(sigma, 1.5), sigma, m.h, m.f};
    R.hk = m.hk;
    R.e = e;
    R.next[0] = m.p0;
    R.next[1] = m.p1;
    R.last[0] = R.last[1] = 0;
    R.t = R.t_last = 0;
    R.dt = 0.01 * a.time_step;
    R.step = 0;
    R.sample = 1;
    R.status = 0;
    if (write) {
        a.mz[e * a.N] = R.next[0] - R.next[1];
        a.time[e * a.N] = 0;
        a.field[e * a.N] = dom_field(a.shape, 0, R.q.h, R.q.f, a.ncomp) * R.hk;
    }
}

// Writes the samples that the accepted step (last, t_last) -> (next, t) has
// passed; false once there are none left.
__device__ inline bool dom_samples(DomRun &R, const DomArgs &a, bool write)
{
    while (R.sample < a.N && !(R.t <= R.sample * a.sampling_time)) {
        if (write) {
            const double mz_last = R.last[0] - R.last[1];
            const double mz_next = R.next[0] - R.next[1];
            const double t_sample = R.sample * a.sampling_time;
            const double beta = (mz_next - mz_last) / (R.t - R.t_last);  // first-order hold
            const int64_t o = R.e * a.N + R.sample;
            a.mz[o] = mz_last + beta * (t_sample - R.t_last);
            a.time[o] = t_sample;
            a.field[o] = dom_field(a.shape, t_sample, R.q.h, R.q.f, a.ncomp) * R.hk;
        }
        R.sample++;
    }
    return R.sample < a.N;
}

__device__ inline void dom_end(DomRun &R, const DomArgs &a)
{
    for (; R.sample < a.N; R.sample++) {  // samples a stopped particle never reached
        const double t_sample = R.sample * a.sampling_time;
        const int64_t o = R.e * a.N + R.sample;
        a.mz[o] = NAN;
        a.time[o] = t_sample;
        a.field[o] = dom_field(a.shape, t_sample, R.q.h, R.q.f, a.ncomp) * R.hk;
    }
    a.status[R.e] = R.status;
    a.steps[R.e] = R.step;
}

// One thread per particle.
__device__ inline void dom_threads(const DomArgs &a, int64_t w)
{
    if (w >= a.E) return;
    DomRun R;
    dom_begin(R, a, a.order ? a.order[w] : w, true);
    const double max_dt = a.end_time / 1000.0;
    const int shape = a.shape;
    const int64_t nc = a.ncomp;
    Rates first = a.N > 1 ? dom_rates(0.0, R.q, shape, nc) : Rates{0, 0};
    while (dom_samples(R, a, true)) {
        R.last[0] = R.next[0];
        R.last[1] = R.next[1];
        R.t_last = R.t;
        if (R.step >= a.max_steps) { R.status = DOM_ST_STEP_LIMIT; break; }
        R.step++;
        double err = 0.0, h = R.dt;
        bool ok = false;
        Rates end;
        for (int attempt = 0; attempt < DOM_MAX_ATTEMPTS && !ok; attempt++) {
            err = dom_trial(R.next, h, R.last, a.time_step, [&](int s) {
                if (s == 0) return first;
                const Rates r = dom_rates(R.t_last + h * stage_time(s), R.q, shape, nc);
                if (s == 4) end = r;
                return r;
            });
            if (err < 1.0) ok = true;
            else h = dom_shorter_step(h, err);
        }
        if (!ok) { R.status = DOM_ST_STEP_LIMIT; break; }
        R.t = R.t_last + h;
        R.dt = dom_next_step(h, err, max_dt);
        if (!isfinite(R.t) || !isfinite(R.dt)) { R.status = DOM_ST_NONFINITE; break; }
        R.dt = R.dt > max_dt ? max_dt : R.dt;
        first = end;
    }
    dom_end(R, a);
}

// Five lanes per particle, six particles per warp: an FP64 instruction takes a
// warp 64 issue cycles however many lanes are active, and the time of a batch
// that leaves sub-partitions idle is that of its longest particle.  The rates
// of a step's stages depend on the time alone, so lane s - 1 evaluates stage
// s = 1..5 (a sine, two exponentials, two divisions) and every lane of the
// particle goes through the same stages with them: one evaluation a trial
// instead of five.  The same operations on the same values.
__device__ inline void dom_lanes(const DomArgs &a, int64_t first_w)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x, group = min(lane / 5, DOM_GROUPS - 1), base = 5 * group;
    const int64_t w0 = first_w + group;
    const int64_t w = w0 < a.lanes ? w0 : a.lanes - 1;  // groups past the end repeat the last one
    const bool write = w0 < a.lanes && lane == base;
    const int stage = min(lane - base, 4) + 1;  // lanes 30 and 31 repeat lane 29
    DomRun R;
    dom_begin(R, a, a.order ? a.order[w] : w, write);
    const double max_dt = a.end_time / 1000.0;
    const int shape = a.shape;
    const int64_t nc = a.ncomp;
    const double hc = stage_time(stage);
    Rates first = dom_rates(0.0, R.q, shape, nc);
    bool alive = dom_samples(R, a, write);
    int attempt = 0;
    double h = R.dt;
    // a pass is one trial of every particle of the warp
    for (;;) {
        if (alive && attempt == 0) {  // a new step
            if (R.step >= a.max_steps) {
                R.status = DOM_ST_STEP_LIMIT;
                alive = false;
            } else {
                R.last[0] = R.next[0];
                R.last[1] = R.next[1];
                R.t_last = R.t;
                R.step++;
                h = R.dt;
            }
        }
        if (!__any_sync(FULL, alive)) break;
        const Rates mine = dom_rates(R.t_last + h * hc, R.q, shape, nc);
        double next[2];
        const double err = dom_trial(next, h, R.last, a.time_step, [&](int s) {
            if (s == 0) return first;
            return Rates{__shfl_sync(FULL, mine.r1, base + s - 1),
                         __shfl_sync(FULL, mine.r2, base + s - 1)};
        });
        const Rates end{__shfl_sync(FULL, mine.r1, base + 3), __shfl_sync(FULL, mine.r2, base + 3)};
        if (!alive) continue;
        R.next[0] = next[0];
        R.next[1] = next[1];
        if (err < 1.0) {
            R.t = R.t_last + h;
            R.dt = dom_next_step(h, err, max_dt);
            if (!isfinite(R.t) || !isfinite(R.dt)) {
                R.status = DOM_ST_NONFINITE;
                alive = false;
                continue;
            }
            R.dt = R.dt > max_dt ? max_dt : R.dt;
            first = end;
            attempt = 0;
            alive = dom_samples(R, a, write);
        } else {
            h = dom_shorter_step(h, err);
            if (++attempt >= DOM_MAX_ATTEMPTS) {
                R.status = DOM_ST_STEP_LIMIT;
                alive = false;
            }
        }
    }
    if (write) dom_end(R, a);
}

// `order` lists particles by expected step count, largest first, so that the
// particles of a warp take similar numbers of steps; the first a.lanes of them
// run five lanes each, the rest one thread each.
__global__ void __launch_bounds__(DOM_THREADS) dom_kernel(DomArgs a)
{
    const int64_t lane_blocks = (a.lanes + DOM_GROUPS - 1) / DOM_GROUPS;
    if (blockIdx.x < lane_blocks) dom_lanes(a, (int64_t)blockIdx.x * DOM_GROUPS);
    else dom_threads(a, a.lanes + (blockIdx.x - lane_blocks) * DOM_THREADS + threadIdx.x);
}

}  // namespace

cudaError_t launch_dom(const DomArgs &a, cudaStream_t stream)
{
    if (a.E == 0) return cudaSuccess;
    const int64_t blocks = (a.lanes + DOM_GROUPS - 1) / DOM_GROUPS +
                           (a.E - a.lanes + DOM_THREADS - 1) / DOM_THREADS;
    dom_kernel<<<(unsigned)blocks, DOM_THREADS, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace magpy
