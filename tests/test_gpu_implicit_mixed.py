"""The mixed-precision implicit midpoint kernel and the launch shape of the
warp-packed FP64 kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cluster(n, seed):
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    return np.full(n, 7e-9), grid * 20e-9 + rng.uniform(-5e-10, 5e-10, (n, 3)), axes


def _args(n, E, steps, dt, implicit=True, seed=3):
    radius, loc, axes = _cluster(n, seed)
    return (E, radius, np.full(n, 2e4), axes, axes.copy(), loc, 4e5, 0.1, 300.0, False, True,
            implicit, dt, dt * (steps - 0.5), 3, np.arange(E) + 5, "sine", 1e4, 3e5, 1e-9)


@pytest.mark.parametrize("n,E", [(1, 3), (2, 1300), (13, 11), (16, 5), (31, 3), (32, 4), (33, 3),
                                 (65, 2)])
def test_mixed_implicit_same_root(gpu_lib, n, E):
    """Both kernels stop within 1e-9 of the norm of the member's first iterate
    (about sqrt(n)/2) of the same root, 2 y - x0 doubles it, and 40 steps add
    up: 40 x 2 x 1e-9 x sqrt(n)/2 each, below 1e-6 for n <= 65; the FP32
    dipolar sum adds about n 6e-8 |h| dt <= 1e-8 a step."""
    from magpy_gb300 import core
    a = core.simulate_ensemble(*_args(n, E, 40, 2e-13), precision="mixed")
    b = core.simulate_ensemble(*_args(n, E, 40, 2e-13), precision="fp64")
    assert np.all(a.status == 0) and np.array_equal(a.steps, b.steps)
    for c in ("mx", "my", "mz"):
        err = np.abs(getattr(a, c)[-1] - getattr(b, c)[-1]).max() / 4e5
        assert err < 1.4e-6, (c, err)


@pytest.mark.parametrize("n", [5, 40])
def test_mixed_implicit_status(gpu_lib, n):
    from magpy_gb300 import _lib, core
    a = core.simulate_ensemble(*_args(n, 3, 4, 2e-13), precision="mixed", max_iter=1)
    assert np.all(a.status & _lib.STATUS_NEWTON_MAXITER)
    assert np.all(np.isfinite(a.mx))


@pytest.mark.parametrize("n,E,implicit", [
    # several lanes per particle, its Newton matrix over 16 or 4 lanes
    (1, 1, True), (1, 1215, True), (1, 1217, True), (2, 607, True), (2, 609, True), (3, 5, True),
    (5, 608, True), (8, 3, True), (1, 1, False), (1, 9729, False), (2, 608, False),
    (3, 609, False), (7, 100, False), (8, 1216, False),
    # past them: one thread per particle
    (8, 609, True), (8, 1217, False), (1, 4865, True), (11, 1300, False), (32, 700, False)])
def test_fp64_launch_shape_is_free(gpu_lib, n, E, implicit):
    """The lanes of a particle, the members of a warp and the warps of a CTA do
    not enter a member's arithmetic: bit-identical trajectories for the
    launcher's choice and for one thread per particle in fully packed warps."""
    from magpy_gb300 import core
    args = _args(n, E, 3, 1e-12 if implicit else 1e-13, implicit)
    a = core.EnsemblePlan(*args).run().arrays()
    b = core.EnsemblePlan(*args).set_launch(4, 0).run().arrays()
    for c in ("mx", "my", "mz", "status", "steps"):
        assert np.array_equal(getattr(a, c), getattr(b, c)), c


@pytest.mark.parametrize("n,implicit", [(1, True), (2, True), (3, True), (8, False)])
def test_fp64_lanes_special_members(gpu_lib, n, implicit):
    """Members beside one that hits the iteration limit, that starts from NaN,
    or without noise and off the field's axis (exact zeros): as with one thread
    per particle."""
    from magpy_gb300 import core
    E = 9
    radius, loc, axes = _cluster(n, 3)
    m0 = np.tile(axes, (E, 1)).reshape(E, n, 3)
    axes = m0.copy()
    m0[1, 0] = np.nan
    axes[2] = m0[2] = [0.0, 0.0, 1.0]
    axes[3] = m0[3] = [-1.0, 0.0, 0.0]
    tile = lambda v: np.concatenate([v] * E)  # noqa: E731
    T = np.full(E, 300.0)
    T[2:4] = 0.0
    for renorm, max_iter in ((False, 1000), (True, 7)):
        args = (E, tile(radius), np.full(E * n, 2e4), axes, m0, tile(loc), 4e5, 0.1, 300.0, renorm,
                True, implicit, 1e-12, 1e-12 * 39.5, 4, np.arange(E), "square", 1e4, 1e10, 1e-9)
        kw = dict(per_member_geometry=True, per_member={"temperature": T}, max_iter=max_iter)
        a = core.EnsemblePlan(*args, **kw).run().arrays()
        b = core.EnsemblePlan(*args, **kw).set_launch(4, 0).run().arrays()
        for c in ("mx", "my", "mz", "status", "steps"):
            np.testing.assert_array_equal(getattr(a, c), getattr(b, c))
        assert a.status[1] & 4 and np.all(a.status[4:] == (1 if implicit and max_iter == 7 else 0))


@pytest.mark.parametrize("n,implicit", [(1, True), (3, False), (33, True)])
@pytest.mark.parametrize("shape", ["sine", "square"])
def test_shared_applied_field(gpu_lib, n, implicit, shape):
    """Lanes compute the applied field of consecutive steps for each other only
    where all members of their warp share it: members beside one of another
    frequency (who compute their own) take the same bits; 70 steps cross a
    block of 32."""
    from magpy_gb300 import core
    E = 40
    args = list(_args(n, E, 70, 1e-12 if implicit else 1e-13, implicit))
    args[16] = shape
    f = np.full(E, 3e5)
    a = core.simulate_ensemble(*args, per_member={"field_frequency": f})
    f[::7] = 4e11  # half periods of 1.25 ps: the square wave turns within the run
    b = core.simulate_ensemble(*args, per_member={"field_frequency": f})
    same = np.repeat(f == 3e5, n)
    for c in ("mx", "my", "mz"):
        assert np.array_equal(getattr(a, c)[:, same], getattr(b, c)[:, same])
        assert not np.array_equal(getattr(a, c)[:, ~same], getattr(b, c)[:, ~same])


@pytest.mark.parametrize("precision,n", [("mixed", 5), ("mixed", 40), ("mixed_tc", 5),
                                         ("mixed_tc", 70)])
def test_no_iteration_with_zero_tolerance(gpu_lib, precision, n):
    """A tolerance of zero stops the reference's iteration before it begins: its
    first iterate is the result.  Two steps of an FP32 dipolar sum (n 6e-8 of
    fields of order 1, times dt 4e-3) differ by below 1e-6."""
    from magpy_gb300 import core
    args = list(_args(n, 3, 3, 2e-13))
    args[-1] = 0.0
    a = core.simulate_ensemble(*args, precision=precision)
    b = core.simulate_ensemble(*args, precision="fp64")
    assert np.all(a.status == 0) and np.all(b.status == 0)
    for c in ("mx", "my", "mz"):
        assert np.abs(getattr(a, c) - getattr(b, c)).max() / 4e5 < 1e-6


@pytest.mark.parametrize("n,E,implicit", [(2, 5, False), (17, 3, True), (33, 3, False)])
def test_device_built_pair_tables(gpu_lib, n, E, implicit):
    """Clusters and temperatures of their own per member: the mixed kernels'
    tables (built on the device from the locations) against the FP64 kernel's
    (from the host).  FP32 tables and sums are off by 6e-8 of fields of order 1,
    over 40 steps of dt <= 4e-3: below 1e-6."""
    from magpy_gb300 import core
    g = core.generate_clusters(E, n, np.arange(E) + 7, packing_fraction=0.3, spacing=2.05)
    args = (E, g["radius"], np.full(E * n, 2e4), g["anisotropy_axis"],
            g["magnetisation_direction"], g["location"], 4e5, 0.1, 300.0, False, True, implicit,
            2e-13, 2e-13 * 39.5, 3, np.arange(E), "constant", 1e4, 0.0, 1e-9)
    kw = dict(per_member_geometry=True, per_member={"temperature": np.linspace(200, 300, E)})
    a = core.simulate_ensemble(*args, precision="mixed", **kw)
    b = core.simulate_ensemble(*args, precision="fp64", **kw)
    for c in ("mx", "my", "mz"):
        err = np.abs(getattr(a, c) - getattr(b, c)).max() / 4e5
        assert 0 < err < 1e-6, err
