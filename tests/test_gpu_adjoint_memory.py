"""What an adjoint object takes of the device's memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_checkpoints_beside_a_run_kept_whole(gpu_lib):
    """64 members of 27 particles, 20000 steps, a checkpoint asked for at every
    step: the run's planes take 1.24e9 bytes, in which form no checkpoint is read
    (0.83e9 bytes of them)."""
    import torch
    from magpy_gb300.adjoint import EnsembleAdjoint
    n, E, steps = 27, 64, 20000
    grid = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2e-8
    axes = np.tile([0.0, 0.0, 1.0], (n, 1))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    adj = EnsembleAdjoint(E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, grid, 4e5, 0.1, 300.0,
                          5e-14, 5e-14 * (steps - 0.5), 5, np.arange(E), "sine", 1e4, 3e9,
                          checkpoint_every=1)
    taken = before - torch.cuda.mem_get_info()[0]
    adj.close()
    assert taken <= 36 * n * E * steps + (64 << 20)
