"""Launch shapes the batch tuner tries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2])
def test_single_particles_and_dimers_have_no_shape_to_tune(gpu_lib, n):
    """Mixed Heun runs of one or two particles ignore the launch shape: the tuner
    times none and reports the default one."""
    from magpy_gb300 import core
    from test_gpu_batch import _group
    rng = np.random.default_rng(3)
    batch = core.EnsembleBatch([_group(n, E, "mixed", rng, 60) for E in (301, 302, 303, 304, 305)],
                               autotune=True)
    try:
        assert [batch.choice(i)[1:3] for i in range(5)] == [(4, 0)] * 5
        assert all(batch.choice(i)[3] > 0 for i in range(5))
    finally:
        batch.close()


@pytest.mark.parametrize("n,E,implicit", [(1, 1000, False), (3, 200, False), (2, 100, True),
                                          (27, 50, False)])
def test_a_reported_shape_is_one_that_a_plan_takes(gpu_lib, n, E, implicit):
    """FP64 groups, small ones run by the launcher's own choice among them: the
    reported shape can be set on a plan of the same ensemble, with the same bits."""
    from magpy_gb300 import core
    from test_gpu_batch import _group
    g = _group(n, E, "fp64", np.random.default_rng(4), 20)
    g["use_implicit"] = implicit
    batch = core.EnsembleBatch([g], autotune=True)
    try:
        prec, bw, mpw, ms = batch.choice(0)
        assert prec == "fp64" and ms > 0
        a = batch.run().groups[0].arrays()
    finally:
        batch.close()
    plan = core.EnsemblePlan(*[g[k] for k in core.EnsembleBatch._POS], g["field_shape"],
                             g["field_amplitude"], g["field_frequency"], precision=prec)
    try:
        b = plan.set_launch(bw, mpw).run().arrays()
    finally:
        plan.close()
    assert np.all(a.status == 0)
    for c in ("mx", "my", "mz"):
        assert np.array_equal(getattr(a, c), getattr(b, c))
