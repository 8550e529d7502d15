"""The adjoint's forms (one member a thread, one with two warps per sum, two
members a thread; with and without the kept dipolar fields) on one ensemble."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(n, copies, steps, every, interactions=True):
    from magpy_gb300.adjoint import EnsembleAdjoint
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    seeds = np.tile([5, 17, 23], copies)
    adj = EnsembleAdjoint(seeds.size, rng.uniform(6e-9, 8e-9, n), np.full(n, 2e4), axes, axes,
                          grid * 20e-9, 4e5, 0.1, 300.0, 5e-14, 5e-14 * (steps - 0.5), 5, seeds,
                          "sine", 1e4, 3e9, interactions, checkpoint_every=every)
    time, field, M = adj.forward()
    _, red = adj.backward(np.array([0.0, 1.0, -2.0, 0.5, 3.0]))
    assert np.all(adj.status == 0)
    adj.close()
    return M, red


@pytest.mark.parametrize("n,copies,steps,every", [
    (1, 6001, 40, 16), (2, 45001, 40, 40), (5, 6401, 40, 7), (13, 1001, 40, 16), (31, 335, 40, 64),
    (32, 335, 40, 16), (33, 201, 40, 16), (64, 201, 20, 16), (27, 6667, 260, 256)])
def test_forms_agree(gpu_lib, n, copies, steps, every):
    """A mean over members does not change when every member is repeated: three
    members (one each a thread; two warps a sum from 5 particles) against a
    large odd number (two a thread from 1000 warps; the last case keeps no
    dipolar fields).  Compared are the device's sensitivities; the gradient's K
    is a difference of three of them.  The forms differ in the order of a split FP32 sum: about
    1e-7 of a field a step, below 5e-5 of the gradients over 260 steps."""
    a, b = _gradient(n, 1, steps, every), _gradient(n, copies, steps, every)
    np.testing.assert_allclose(a[0], b[0], rtol=1e-5, atol=1e-6 * np.abs(a[0]).max())
    for x, y in zip(a[1:], b[1:]):
        np.testing.assert_allclose(x, y, rtol=5e-5)


def test_forms_agree_without_interactions(gpu_lib):
    a, b = _gradient(8, 1, 40, 16, False), _gradient(8, 3001, 40, 16, False)
    for x, y in zip(a[1:], b[1:]):
        np.testing.assert_allclose(x, y, rtol=5e-5)


@pytest.mark.parametrize("steps,every", [(1100, 256), (1100, 1000)])
def test_whole_run_and_segments_agree(gpu_lib, steps, every):
    """The fields of the whole run kept by the forward pass (2049 members) or of a
    segment by its recomputation (4098 members, 4.4 GB for the whole run): the same
    members twice as often, the same bits of each member's sensitivities, their
    double-precision sums in another order."""
    a, b = _gradient(27, 683, steps, every), _gradient(27, 1366, steps, every)
    np.testing.assert_allclose(a[0], b[0], rtol=1e-11)
    for x, y in zip(a[1:], b[1:]):
        np.testing.assert_allclose(x, y, rtol=1e-9)
