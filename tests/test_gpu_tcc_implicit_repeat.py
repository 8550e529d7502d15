"""The cluster implicit kernel reads a step's first member tile only when every
CTA of the cluster has written it: repeated runs give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E,nb", [(20, 33, 32), (84, 70, 64), (85, 41, 40), (200, 40, 40)])
def test_repeated_runs_are_identical(gpu_lib, n, E, nb):
    from magpy_gb300 import core
    rng = np.random.default_rng(n)
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    loc = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    plan = core.EnsemblePlan(E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, loc, 4e5, 0.05,
                             300.0, False, True, True, 2e-13, 2e-13 * 70.5, 4, np.arange(E) + 3,
                             "sine", 1e4, 3e9, precision="mixed_tc").set_launch(4, nb)
    a = plan.run().arrays()
    assert np.all(a.status == 0)
    for _ in range(3):
        b = plan.run().arrays()
        for c in ("mx", "my", "mz"):
            assert np.array_equal(getattr(a, c), getattr(b, c))


@pytest.mark.parametrize("nb", [32, 40, 64])
@pytest.mark.parametrize("n,E", [(2, 3), (41, 33), (42, 64), (43, 41), (85, 2), (126, 65)])
def test_forms_match_fp64(gpu_lib, n, E, nb):
    """Against the FP64 kernel, at the edges of a CTA's 42 particles and of the
    member tiles.  Both stop within 1e-9 of the norm of the member's first iterate
    (below sqrt(n)) of their roots, 2 y - x0 doubles it: 2e-9 sqrt(126) a step each;
    the field's 2e-6 of dt |h| below 0.1 adds 2e-7: 20 steps below 5e-6."""
    from magpy_gb300 import core
    rng = np.random.default_rng(n + E)
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    loc = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    args = (E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, loc, 4e5, 0.05, 300.0, False, True,
            True, 2e-13, 2e-13 * 19.5, 3, np.arange(E) + 3, "sine", 1e4, 3e9)
    a = core.EnsemblePlan(*args, precision="mixed_tc").set_launch(4, nb).run().arrays()
    b = core.simulate_ensemble(*args, precision="fp64")
    assert np.all(a.status == 0) and np.array_equal(a.steps, b.steps)
    for c in ("mx", "my", "mz"):
        assert np.abs(getattr(a, c) - getattr(b, c)).max() <= 5e-6 * 4e5


@pytest.mark.parametrize("precision", ["mixed", "mixed_tc"])
@pytest.mark.parametrize("dt,tilt", [(2e-13, 0.0), (2e-13, 1e-40), (1e-55, 0.0), (1e-55, 0.3)])
def test_stage_map_outside_the_integer_range(gpu_lib, precision, dt, tilt):
    """Components that are zero or tiny, and steps so small that dt h is below the
    integer products' range, take the plain products: the FP64 kernel's result to
    the solver's tolerance (2e-9 sqrt(2) a step; 9 steps)."""
    from magpy_gb300 import core
    m0 = np.array([[tilt, 0.0, 1.0], [0.0, tilt, -1.0]])
    m0 /= np.linalg.norm(m0, axis=1, keepdims=True)
    args = (3, np.full(2, 7e-9), np.full(2, 2e4), np.array([[1.0, 0, 0], [0, 1.0, 0]]), m0,
            np.array([[0.0, 0, 0], [2e-8, 0, 0]]), 4e5, 0.1, 0.0, False, True, True, dt, dt * 9.5,
            3, np.arange(3), "constant", 1e4, 0.0)
    a = core.simulate_ensemble(*args, precision=precision)
    b = core.simulate_ensemble(*args, precision="fp64")
    assert np.all(a.status == 0)
    for c in ("mx", "my", "mz"):
        assert np.abs(getattr(a, c) - getattr(b, c)).max() <= 1e-7 * 4e5
