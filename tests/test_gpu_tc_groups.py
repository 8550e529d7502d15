"""The tensor-core Heun kernel's member groups: 8 to 32 members of a CTA in two
groups of 4 to 16, chosen from the ensemble size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152


def _plan(core, n, E):
    rng = np.random.default_rng(n)
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    loc = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    return core.EnsemblePlan(E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, loc, 4e5, 0.1, 300.0,
                             False, True, False, 5e-14, 5e-14 * 39.5, 3, np.arange(E) + 7, "sine",
                             1e4, 3e10, precision="mixed_tc")


# members per CTA the rule takes: 8 at E <= 8 x 152, 12, 16, .. 28, then 32
@pytest.mark.parametrize("n", [2, 7, 33, 64])
@pytest.mark.parametrize("E", [1, 8 * SMS - 1, 8 * SMS + 1, 12 * SMS, 16 * SMS - 3, 20 * SMS - 5,
                               24 * SMS, 28 * SMS - 9, 28 * SMS + 1, 32 * SMS + 1])
def test_group_sizes_agree(gpu_lib, n, E):
    """A member's arithmetic does not depend on its place in a group: the groups
    the rule takes give the bits that 32 members a CTA give."""
    from magpy_gb300 import core
    plan = _plan(core, n, E)
    a = plan.run().arrays()
    b = plan.set_launch(1).run().arrays()
    assert np.all(a.status == 0) and np.array_equal(a.steps, b.steps)
    for c in ("mx", "my", "mz"):
        x = getattr(a, c)
        assert np.all(np.isfinite(x)) and np.array_equal(x, getattr(b, c))
    m = np.stack([a.mx[-1], a.my[-1], a.mz[-1]], 1)
    assert len(np.unique(m, axis=0)) == len(m)   # no member left out or done twice
