"""Rounding errors of the mixed Heun kernels, read from the float-float state,
against those of a statement of the step in numpy: field, drift (lib/llg.cpp:14-29)
and diffusion (:92-106) in FP32 with each product-sum fused once, and an
error-free addition of the FP32 increment to the state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F, D = np.float32, np.float64


def _fma(a, b, c):
    """a b + c rounded once to FP32 (the FP64 product is exact)."""
    return (a.astype(D) * b.astype(D) + c.astype(D)).astype(F)


def _drift(m, alpha, h, fma):
    o = []
    for c in range(3):
        v, w = (c + 1) % 3, (c + 2) % 3
        cr = fma(m[w], h[v], -(m[v] * h[w]))
        s, q = fma(m[v], m[v], m[w] * m[w]), fma(m[v], h[v], m[w] * h[w])
        o.append(fma(alpha, fma(h[c], s, -(m[c] * q)), cr))
    return o


def _run(m0, ax, sr, alpha, happ, dt, w, T):
    """States after the steps of w [steps][3][items] in the arithmetic of type T;
    alpha [items].  T = FP32: (hi + lo) in FP64."""
    fma = _fma if T is F else (lambda a, b, c: a * b + c)
    cast = lambda a: np.asarray(a, T)  # noqa: E731
    hi, lo = [cast(m) for m in m0], [np.zeros_like(cast(m)) for m in m0]
    ax, sr, alpha, dt, sq = [cast(a) for a in ax], cast(sr), cast(alpha), cast(dt), cast(np.sqrt(dt))
    dt, sq = np.full_like(hi[0], dt), np.full_like(hi[0], sq)
    half = T(0.5)

    def field(m):
        d = fma(m[2], ax[2], fma(m[1], ax[1], m[0] * ax[0]))
        return [d * ax[0], d * ax[1], fma(d, ax[2], np.full_like(d, happ))]

    for k in range(w.shape[0]):
        wk = [cast(w[k, c]) for c in range(3)]
        noise = lambda m: [sr * g for g in _drift(m, alpha, wk, fma)]  # noqa: E731
        a, b = _drift(hi, alpha, field(hi), fma), noise(hi)
        xt = [hi[c] + fma(dt, a[c], sq * b[c]) for c in range(3)]
        ta, tb = _drift(xt, alpha, field(xt), fma), noise(xt)
        for c in range(3):
            d = fma(half * dt, a[c] + ta[c], half * sq * (b[c] + tb[c]))
            s = hi[c] + d
            v = s - hi[c]
            e = (hi[c] - (s - v)) + (d - v) + lo[c]
            hi[c], lo[c] = s + e, e - ((s + e) - s)
    return np.stack([h.astype(D) + l.astype(D) for h, l in zip(hi, lo)])


def _inputs(items, steps, thermal, seed):
    """Parameters that FP32 holds, so that errors are those of the steps."""
    rng = np.random.default_rng(seed)
    unit = lambda v: (v / np.linalg.norm(v, axis=0)).astype(F).astype(D)  # noqa: E731
    ax, m0 = unit(rng.normal(size=(3, items))), unit(rng.normal(size=(3, items)))
    sr = (thermal * np.exp(0.15 * rng.normal(size=items))).astype(F).astype(D)
    w = rng.normal(size=(steps, 3, items)).astype(F).astype(D)
    return ax, m0, sr, w


def _gpu(n, ax, m0, sr, alpha, happ, dt, w):
    """The same from the mixed kernel, n particles that do not interact a call."""
    from magpy_gb300 import core
    steps, _, items = w.shape
    out = np.empty((3, items))
    pad = np.zeros((1, n, 3))  # the sample holds the state before the last step
    for i in range(0, items, n):
        s = slice(i, i + n)
        noise = np.concatenate([w[:, :, s].transpose(0, 2, 1), pad])
        r = core.simulate_reduced(n, sr[s], np.ones(n), np.ones(n), ax[:, s].T, m0[:, s].T,
                                  np.zeros((n, n, 3)), np.ones((n, n)), "constant", happ, 1.0,
                                  2e4, 1.0, alpha, 1.0, dt, (steps + 0.5) * dt, noise.ravel(),
                                  False, False, False, 1e-9, 2, precision="mixed")
        assert r["status"] == 0 and r["steps"] == steps + 1
        out[:, s] = np.stack([r[c][:, 1] for c in "xyz"])
    return out


def _rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2)))


@pytest.mark.parametrize("n,items", [(1, 1500), (2, 3000)])
def test_increments_are_added_to_the_state_without_error(gpu_lib, n, items):
    """Single particles and dimers in noise, alpha = 0.1.  Adding an increment to
    the state's low word first rounds to 2^-25 of the increment and raises the
    error by 6 % or more; the statement's own spread over this many items is
    below 1 %."""
    alpha, happ, dt, steps = float(F(0.1)), 0.125, 2.0 ** -10, 300
    ax, m0, sr, w = _inputs(items, steps, 0.11, 31)
    al = np.full(items, alpha)
    exact = _run(m0, ax, sr, al, happ, dt, w, D)
    stated = _rms(_run(m0, ax, sr, al, happ, dt, w, F), exact)
    assert _rms(_gpu(n, ax, m0, sr, alpha, happ, dt, w), exact) <= 1.03 * stated


@pytest.mark.parametrize("n", [1, 2, 30, 500, 1000])
def test_the_stage_map_forms_no_terms_that_cancel(gpu_lib, n):
    """T = 0 and alpha = 1, where the damping term's rounding is what there is:
    expanded to v |m|^2 - m (m.v) it has terms that cancel, and the error is 1.4
    times the statement's."""
    items, happ, dt, steps = max(1000, n), 0.125, 2.0 ** -10, 300
    ax, m0, sr, w = _inputs(items // n * n, steps, 0.0, 32)
    al = np.ones(m0.shape[1])
    exact = _run(m0, ax, sr, al, happ, dt, w, D)
    stated = _rms(_run(m0, ax, sr, al, happ, dt, w, F), exact)
    assert _rms(_gpu(n, ax, m0, sr, 1.0, happ, dt, w), exact) <= 1.1 * stated


@pytest.mark.parametrize("n,mpc", [(200, 2), (200, 4), (320, 2), (320, 4)])
def test_the_map_with_several_members_a_block(gpu_lib, n, mpc):
    """The same for clusters of more than 32 particles that share their
    parameters, several members a CTA; the time step and field in SI units are
    those that reduce to the statement's."""
    from magpy_gb300 import core
    E, steps, ms, K, happ, dt = 5, 300, 4e5, 2e4, 0.125, 2.0 ** -10
    ax, m0, sr, w = _inputs(n, steps, 0.0, 34)
    exact = _run(m0, ax, sr, np.ones(n), happ, dt, w, D)
    stated = _rms(_run(m0, ax, sr, np.ones(n), happ, dt, w, F), exact)
    # lib/simulation.cpp:519-549
    mu0, gyro = 1.25663706e-6, 1.76086e11
    hk = 2 * K / mu0 / ms
    dt_si = dt * 2 / (gyro * mu0 * hk)
    plan = core.EnsemblePlan(E, np.full(n, 7e-9), np.full(n, K), ax.T, m0.T, np.zeros((n, 3)), ms,
                             1.0, 0.0, False, False, False, dt_si, (steps + 0.5) * dt_si, 2,
                             np.arange(E), "constant", happ * hk, precision="mixed")
    try:
        a = plan.set_launch(4, mpc).run().arrays()
    finally:
        plan.close()
    assert np.all(a.status == 0) and np.all(a.steps == steps + 1)
    got = np.stack([a.mx[1], a.my[1], a.mz[1]]).reshape(3, E, n) / ms
    for e in range(E):
        assert _rms(got[:, e], exact) <= 1.1 * stated
