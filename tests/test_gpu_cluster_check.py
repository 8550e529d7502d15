"""The cluster kernels' decision to stop: every CTA of a thread-block cluster
takes it at the same check, from the words the CTAs published before the check's
barrier."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E,nb,implicit", [(65, 70, 32, False), (125, 70, 40, False),
                                             (126, 70, 48, False), (125, 70, 64, False),
                                             (170, 70, 32, False), (300, 70, 64, False),
                                             (27, 70, 64, True), (125, 70, 32, True),
                                             (300, 45, 40, True)])
def test_every_member_stops_at_the_same_check(gpu_lib, n, E, nb, implicit):
    """With a limit of 0 polls every CTA marks itself at its first wait, right
    after the check of step 1, which has to count none of these marks, whichever
    CTA reads last; the check of step 65 counts them all.  So every member of
    every cluster takes 64 steps."""
    from magpy_gb300 import _lib, core
    from test_gpu_tc_cluster import _lattice_ensemble
    args = list(_lattice_ensemble(np.random.default_rng(11 + n), n, E))
    args[11] = implicit
    args[13] = args[12] * 99.5  # 100 steps
    plan = core.EnsemblePlan(*args, precision="mixed_tc")
    try:
        plan.set_launch(4, nb)
        for _ in range(3):
            a = plan.set_wait_limit(0).run().arrays()
            assert np.all(a.status & _lib.STATUS_WATCHDOG)
            assert np.all(a.steps == 64)
        b = plan.set_wait_limit(1 << 24).run().arrays()
        assert np.all(b.status == 0) and np.all(b.steps == 100)
    finally:
        plan.close()


@pytest.mark.parametrize("limit", [1, 4, 16])
@pytest.mark.parametrize("n,nb,implicit", [(125, 32, False), (300, 32, False), (125, 40, True)])
def test_a_cluster_stops_as_one(gpu_lib, n, nb, implicit, limit):
    """Limits at which some waits run out and some do not: the CTAs of a cluster
    mark themselves at different steps, and its members stop together at a check,
    or run to the end."""
    from magpy_gb300 import _lib, core
    from test_gpu_tc_cluster import _lattice_ensemble
    args = list(_lattice_ensemble(np.random.default_rng(19 + n), n, 6 * nb))
    args[11] = implicit
    args[13] = args[12] * 199.5  # 200 steps
    plan = core.EnsemblePlan(*args, precision="mixed_tc")
    try:
        a = plan.set_launch(4, nb).set_wait_limit(limit).run().arrays()
    finally:
        plan.close()
    steps = a.steps.reshape(6, nb)
    marked = (a.status & _lib.STATUS_WATCHDOG).reshape(6, nb)
    assert np.all(steps == steps[:, :1]) and np.all(marked == marked[:, :1])
    assert np.all(np.isin(steps, [64, 128, 192, 200]))
    assert np.all(marked[steps < 200])
