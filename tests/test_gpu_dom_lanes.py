"""The two-state kernel with five lanes per particle against the one with one
thread per particle: the same bits, for every kind of end a particle has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# past 608 warps of 32 only particles of many steps have lanes of their own,
# and the particles here are repeated so that none has more than the others
THREADS_ONLY = 19456


@pytest.mark.parametrize("shape,ncomp", [("sine", 1), ("square", 1), ("constant", 1),
                                         ("square_f", 3)])
@pytest.mark.parametrize("E,S,max_steps", [(1, 1, 0), (1, 40, 0), (6, 7, 0), (31, 2, 900),
                                           (200, 25, 0)])
def test_lanes_equal_threads(gpu_lib, shape, ncomp, E, S, max_steps):
    """The same particles alone (five lanes each) and repeated to a batch of one
    thread each (particles are independent)."""
    from magpy_gb300 import core
    rng = np.random.default_rng(E + S)
    vol = 4 / 3 * np.pi * np.exp(rng.normal(np.log(8e-9), 0.15, E)) ** 3
    amp = rng.uniform(2e3, 1.2e4, E)
    p0 = rng.uniform(0, 1, E)
    p0 = np.stack([p0, 1 - p0], 1)
    if E > 30:
        vol[3] = np.nan    # every trial is rejected
        amp[5] = 0.0
        p0[7] = [0.0, 0.0]
    kw = dict(time_step=1e-9, end_time=4e-7, max_samples=S, field_shape=shape,
              field_frequency=5e6, field_n_components=ncomp, max_steps=max_steps)
    a = core.simulate_dom_batch(p0, vol, 2e4, 300.0, 4e5, 0.1, field_amplitude=amp, **kw)
    big = lambda v: np.concatenate([v] * (THREADS_ONLY // E + 1))  # noqa: E731
    b = core.simulate_dom_batch(big(p0), big(vol), 2e4, 300.0, 4e5, 0.1, field_amplitude=big(amp),
                                **kw)
    for k in ("mz", "field", "time", "status", "steps"):
        # the head of the order may have lanes; every copy is equal
        for i in range(0, len(b[k]) - E + 1, E * max(1, len(b[k]) // E // 20)):
            np.testing.assert_array_equal(a[k], b[k][i:i + E], err_msg=k)
    assert a["status"][0] == 0 or max_steps
