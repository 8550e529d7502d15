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
