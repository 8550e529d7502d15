"""The FP64 pair sum with its products by integer multiplies: the oracle's bits
for zeros, for magnitudes at the ends of the range it takes, and past them
(where the FP64 products are used)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 33, 64])
@pytest.mark.parametrize("implicit", [False, True])
@pytest.mark.parametrize("form", ["lattice", "tiny", "tinier", "near", "nearer", "weak"])
def test_pair_sum_range(gpu_lib, oracle, n, implicit, form):
    from magpy_gb300 import core
    from oracle.pyoracle import reduced_inputs
    rng = np.random.default_rng(n + 100 * implicit)
    inp = reduced_inputs(rng, n)
    inp["v_red"] = np.round(inp["v_red"], 1)
    if form == "lattice":  # exact zeros in moments, axes and unit vectors; no noise
        side = int(np.ceil(n ** (1 / 3)))
        pts = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        vec = 2.0 * (pts[None] - pts[:, None])
        inp["dist_mag"] = np.sqrt((vec ** 2).sum(-1))
        with np.errstate(invalid="ignore"):
            inp["unit_dist"] = vec / inp["dist_mag"][..., None]
        inp["m0"] = np.tile([0.0, 0.0, 1.0], (n, 1))
        inp["m0"][::3] = [-1.0, 0.0, -0.0]
        inp["axes"] = np.abs(inp["m0"])[:, [2, 1, 0]]
        inp["sr"] = np.zeros(n)
    elif form in ("tiny", "tinier"):  # 2^-80 is the smallest the products take
        inp["m0"][:, 0] = (2.0 ** -80 if form == "tiny" else 2.0 ** -81) * (1 + 2.0 ** -40)
        inp["sr"][:] = 0.0
    elif form in ("near", "nearer"):  # pair factors about 2^30 and 2^60
        inp["dist_mag"] = inp["dist_mag"] * (2.0 ** -10 if form == "near" else 2.0 ** -20)
        inp["m0"] *= 2.0 ** -12
    else:  # pair factors below 2^-80
        inp["dist_mag"] = inp["dist_mag"] * 2.0 ** 28
    dt, S = 1e-3 if form not in ("near", "nearer") else 1e-12, 4
    end = dt * 8.5
    K = core.step_count(dt, end, S)
    noise = rng.normal(size=K * 3 * n)
    kw = dict(field_shape="constant", happ=0.3, fapp=0.0, dt=dt, end_time=end, max_samples=S,
              use_implicit=implicit, renorm=False, interactions=True)
    g = core.simulate_reduced(n, inp["sr"], inp["k_red"], inp["v_red"], inp["axes"], inp["m0"],
                              inp["unit_dist"], inp["dist_mag"], "constant", 0.3, 0.0, 2e4, 1.0,
                              0.1, 4e5, dt, end, noise, False, True, implicit, 1e-9, S, max_iter=60)
    o = oracle.full_dynamics_reduced(inp, noise=noise, max_iter=60, **kw)
    for c in "xyz":
        np.testing.assert_array_equal(g[c], o[c])
    assert np.all(np.isfinite(g["x"][:, :2]))  # the strongest coupling blows up later
