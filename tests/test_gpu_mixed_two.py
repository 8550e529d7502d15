"""The mixed Heun kernel with two particles per thread (a dimer, or two members
of one particle each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E", [(1, 1), (1, 2), (1, 65), (1, 20001), (2, 1), (2, 33), (2, 77825)])
@pytest.mark.parametrize("form", ["sine", "renorm", "noise", "free"])
def test_two_per_thread_strong_error(gpu_lib, n, E, form):
    """Against the FP64 kernel on the same increments.  A step's FP32 rounding is
    6e-8 of increments below 0.1: 30 steps are below 30 x 6e-9, and the
    renormalisation's FP32 factor adds 30 x 1.2e-7 of the unit moment."""
    from magpy_gb300 import core
    rng = np.random.default_rng(E)
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    steps, dt = 31, 1e-13
    noise = rng.normal(size=(E, steps * 3 * n)) if form == "noise" and E < 1000 else None
    args = (E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, np.arange(3 * n).reshape(n, 3) * 1e-8,
            4e5, 0.1, 300.0, form == "renorm", form != "free", False, dt, dt * (steps - 0.5), 3,
            np.arange(E) + 3, "sine" if form == "sine" else "constant", 1e4, 3e10)
    kw = dict(noise=noise, per_member={"temperature": np.linspace(250, 350, E)})
    a = core.simulate_ensemble(*args, precision="mixed", **kw)
    b = core.simulate_ensemble(*args, precision="fp64", **kw)
    assert np.all(a.status == 0) and np.array_equal(a.steps, b.steps)
    for c in ("mx", "my", "mz"):
        assert np.abs(getattr(a, c) - getattr(b, c)).max() / 4e5 < 4e-6
        np.testing.assert_allclose(getattr(a, c)[0], getattr(b, c)[0], rtol=1e-13)


@pytest.mark.parametrize("n", [1, 2])
def test_two_per_thread_status(gpu_lib, n):
    """A member that starts from NaN is reported, and leaves its neighbours alone."""
    from magpy_gb300 import core
    E = 5
    m0 = np.zeros((E, n, 3))
    m0[..., 2] = 1.0
    def run(m):
        return core.simulate_ensemble(
            E, np.full(E * n, 7e-9), np.full(E * n, 2e4), np.tile([0, 0, 1.0], (E * n, 1)),
            m.reshape(-1, 3), np.tile(np.arange(3 * n) * 1e-8, E), 4e5, 0.1, 300.0, False, True,
            False, 1e-13, 1e-13 * 9.5, 3, np.arange(E), per_member_geometry=True,
            precision="mixed")
    a = run(m0)
    bad = m0.copy()
    bad[2, 0, 1] = np.nan
    b = run(bad)
    assert list(b.status) == [0, 0, 4, 0, 0]
    keep = np.repeat(np.arange(E) != 2, n)
    for c in ("mx", "my", "mz"):
        assert np.array_equal(getattr(a, c)[:, keep], getattr(b, c)[:, keep])


@pytest.mark.parametrize("renorm", [False, True])
def test_one_or_two_members_per_thread_agree(gpu_lib, renorm):
    """Single particles: one member a thread up to 32 x 4 x 152 members, two above;
    the same bits."""
    from magpy_gb300 import core
    one = np.ones(1)
    def run(E):
        return core.simulate_ensemble(
            E, 7e-9 * one, 2e4 * one, np.array([[0, 0.6, 0.8]]), np.array([[1.0, 0, 0]]),
            np.zeros((1, 3)), 4e5, 0.1, 300.0, renorm, False, False, 1e-13, 1e-13 * 30.5, 3,
            np.arange(E), "sine", 1e4, 3e10, precision="mixed")
    a, b = run(32 * 4 * 152), run(32 * 4 * 152 + 1)
    assert np.all(a.status == 0) and np.all(b.status == 0)
    for c in ("mx", "my", "mz"):
        assert np.array_equal(getattr(a, c), getattr(b, c)[:, :-1])
