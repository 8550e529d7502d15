"""What a plan takes of the device's memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_resident_cluster_plans_have_no_exchange_buffers(gpu_lib):
    """126 particles, 65536 members, one sample: eight rows of inputs and three of
    outputs, FP64 a particle, and a record a member.  (The exchange buffers, which
    the kernel that holds D in tensor memory does not read, were 201 MB more.)"""
    import torch
    from magpy_gb300 import core
    n, E = 126, 65536
    grid = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2e-8
    axes = np.tile([0.0, 0.0, 1.0], (n, 1))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = core.EnsemblePlan(E, np.full(n, 7e-9), np.full(n, 2e4), axes, axes, grid, 4e5, 0.1,
                             300.0, False, True, False, 5e-14, 5e-13, 1, np.arange(E),
                             precision="mixed_tc")
    taken = before - torch.cuda.mem_get_info()[0]
    plan.close()
    assert taken <= 8 * (11 * n + 32) * E + (64 << 20)
