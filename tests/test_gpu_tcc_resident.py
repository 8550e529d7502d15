"""The cluster Heun kernel for 65 to 126 particles (two or three CTAs a cluster, two member groups,
the moments of a member tile in every CTA's shared memory)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [32, 40, 48, 64])
@pytest.mark.parametrize("n,E", [(65, 1), (83, 33), (84, 64), (85, 65), (125, 41), (126, 97)])
def test_resident_forms_match_fp64(gpu_lib, n, E, nb):
    """Against the FP64 kernel on the same increments, at the edges of the CTAs'
    42 particles and of the member tiles.  A step's FP32 rounding is 6e-8 of
    increments below 0.1 and the field's error 2e-6 of them: 40 steps stay below
    40 x 0.1 x 2.1e-6 of the unit moment."""
    from magpy_gb300 import core
    rng = np.random.default_rng(n + E)
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    loc = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    args = (E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, loc, 4e5, 0.1, 300.0, False, True,
            False, 5e-14, 5e-14 * 39.5, 3, np.arange(E) + 11, "sine", 1e4, 3e10)
    a = core.EnsemblePlan(*args, precision="mixed_tc").set_launch(4, nb).run().arrays()
    b = core.simulate_ensemble(*args, precision="fp64")
    assert np.all(a.status == 0) and np.array_equal(a.steps, b.steps)
    for c in ("mx", "my", "mz"):
        assert np.abs(getattr(a, c) - getattr(b, c)).max() <= 8.4e-6 * 4e5


@pytest.mark.parametrize("n", [33, 64, 70, 126])
def test_failed_member_and_single_sample(gpu_lib, n):
    """A member whose injected increments hold a NaN is reported and leaves the
    members of its group and of the other one alone; a run of one sample takes no
    step."""
    from magpy_gb300 import core
    E, steps = 21, 70
    m0 = np.zeros((n, 3))
    m0[:, 2] = 1.0
    loc = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    noise = np.random.default_rng(n).normal(size=(E, steps * 3 * n))
    def run(samples, noise):
        return core.simulate_ensemble(
            E, np.full(n, 7e-9), np.full(n, 2e4), m0, m0, loc, 4e5, 0.1, 300.0, False, True, False,
            5e-14, 5e-14 * (steps - 0.5), samples, np.arange(E) + 11, "sine", 1e4, 3e10,
            precision="mixed_tc", noise=noise)
    a, one = run(3, noise), run(1, noise)
    assert np.all(a.status == 0) and np.all(one.status == 0) and np.all(one.steps == 0)
    np.testing.assert_array_equal(one.mz[0], a.mz[0])
    bad = noise.copy()
    bad[5, 3 * n * 2 + 4] = np.nan
    b = run(3, bad)
    assert list(np.nonzero(b.status)[0]) == [5] and b.status[5] == 4
    keep = np.repeat(np.arange(E) != 5, n)
    for c in ("mx", "my", "mz"):
        assert np.array_equal(getattr(a, c)[:, keep], getattr(b, c)[:, keep])
