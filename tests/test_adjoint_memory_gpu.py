"""Device memory that gradients keep between calls: bounded over all grids of
the process, and given back on request."""

import gc

import numpy as np
import pytest

from gpu_helpers import smooth_eps, to_np

pytestmark = pytest.mark.gpu

STEPS = 900  # 96^3 with 10 CPML layers: 15.5 MB a snapshot, 14 GB for all of them


def test_kept_snapshots_bounded_and_released(cuda):
    import torch

    from jaxphys_b200 import ConfigurationError, EMGrid3D, PointSource3D
    from jaxphys_b200.em.adjoint import probe_traces

    size = (96, 96, 96)
    eps = torch.tensor(smooth_eps(size, 1.0, 4.0, seed=1), dtype=torch.float32, device=cuda)

    def grid():
        g = EMGrid3D(size=size, resolution=1.0, boundary="cpml", pml_layers=10)
        g.add_source(PointSource3D(frequency=0.05 / g.default_dt(), position=(40, 48, 48)))
        g.add_probe((56, 48, 50), "ez")
        g.prepare()
        return g

    def grad(g):
        e = eps.clone().requires_grad_(True)
        (probe_traces(g, e, STEPS) ** 2).sum().backward()
        return to_np(e.grad)

    def used():
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, total = torch.cuda.mem_get_info(0)
        return total - free, total

    grids = [grid() for _ in range(6)]
    start, total = used()
    if total - start < 96 << 30:
        pytest.skip("needs 96 GB free")
    want = grad(grids[0])
    one = used()[0] - start
    for g in grids[1:5]:
        g.adjoint_forward(STEPS)
    assert np.array_equal(grad(grids[5]), want) and np.abs(want).max() > 0
    held = used()[0] - start
    # beside the snapshots: checkpoints, a segment's snapshots and adjoint
    # fields, below 2 GB a grid (30 checkpoints of 31 MB, 30 snapshots)
    assert held < total // 4 + 6 * (2 << 30), (one, held)
    grids[0].adjoint_release()
    left = used()[0] - start
    assert one > 8 << 30 and left < held - one + (1 << 30), (one, held, left)
    with pytest.raises(ConfigurationError, match="adjoint_forward first"):
        grids[0].adjoint_backward(torch.zeros((STEPS, 1), device=cuda))
    assert np.array_equal(grad(grids[0]), want)
