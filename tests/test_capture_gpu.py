"""A grid's first steps captured into a caller's CUDA graph, without a step
before: no allocation, copy from the host or synchronisation in them where
the grid has nothing to tune.  Replayed, the graph gives what the same call
gives outside one."""

import numpy as np
import pytest

from gpu_helpers import grid_fields, to_np

pytestmark = pytest.mark.gpu

STEPS = 6


def _capture_and_replay(step):
    import torch

    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        step()
    graph.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize("size,boundary,sources", [
    ((13, 12, 11), "cpml", 3), ((12, 14, 10), "absorbing", 3), ((16, 12, 20), "periodic", 3),
    ((16, 16, 16), "absorbing", 0)])
def test_first_steps_of_a_3d_grid(cuda, size, boundary, sources):
    from jaxphys_b200 import EMGrid3D, PointSource3D
    from jaxphys_b200 import _native as nat

    def grid():
        g = EMGrid3D(size=size, resolution=1.0, boundary=boundary, pml_layers=3)
        for i in range(sources):
            g.add_source(PointSource3D(frequency=0.05 / g.default_dt(), position=(5 + i, 6, 5)))
        g.prepare()
        if sources:
            g._ensure_waves(STEPS)
        g.set_field("ey", np.random.default_rng(0).standard_normal(size).astype(np.float32))
        return g

    def step(g):
        nat.check(nat.load().jxf_grid3d_step(g._h, STEPS, None, nat.stream_handle()), "step")

    g, ref = grid(), grid()
    _capture_and_replay(lambda: step(g))
    step(ref)
    for a, b in zip(grid_fields(g), grid_fields(ref)):
        assert np.array_equal(a, b) and np.abs(b).max() > 0
