"""The stopping norm of the tensor-core implicit kernel for an update whose square
is past FP32's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_huge_update_does_not_stop_a_member_as_converged(gpu_lib):
    """Two particles too far apart to interact, the first nearly along z in the
    noise's own direction with alpha v m = -2, all powers of two: the first
    iteration's FP32 Jacobian is [[0, b/2, -2e], [-b/2, 0, 0], [4e, 0, 1]] with
    b = -2^-79 and e = 1e-4, so the update's y is 1e-4 * 2^80 = 1.2e20, whose
    square FP32 does not hold.  The member has not converged: it goes on (its FP16
    moments overflow then), and reports what becomes of it."""
    from magpy_gb300 import core
    n, dt, eps = 2, 2.0 ** -10, 1e-4
    m0 = np.array([[eps, 0, 1.0], [0, 0, 1.0]])
    axes = np.array([[0, 1.0, 0], [0, 1.0, 0]])
    unit = np.zeros((n, n, 3))
    unit[0, 1], unit[1, 0] = [0, 0, 1], [0, 0, -1]
    noise = np.zeros((2, n, 3))
    noise[0, 0, 2] = -(2.0 ** -79) / np.sqrt(dt)
    r = core.simulate_reduced(n, np.ones(n), np.zeros(n), np.ones(n), axes, m0, unit,
                              np.full((n, n), 1e6), "constant", 0.0, 1.0, 2e4, 1.0, 2.0 ** 80,
                              4e5, dt, 0.5 * dt, noise.ravel(), False, True, True, 1e-9, 2,
                              precision="mixed_tc")
    assert r["steps"] == 1
    assert r["status"] != 0
