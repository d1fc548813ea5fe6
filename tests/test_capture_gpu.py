"""A grid's first steps captured into a caller's CUDA graph, without a step
before: no allocation, copy from the host or synchronisation in them where
the grid has nothing to tune.  Replayed, the graph gives what the same call
gives outside one."""

import numpy as np
import pytest

from gpu_helpers import grid_fields

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


@pytest.mark.parametrize("boundary", ["absorbing", "periodic", "reflecting"])
def test_first_steps_of_a_2d_grid(cuda, boundary):
    """And the steps after those, outside a graph: several per launch."""
    from jaxphys_b200 import EMGrid, PlaneWave, Wall
    from jaxphys_b200 import _native as nat

    lib = nat.load()

    def grid():
        g = EMGrid(size=(37, 45), boundary=boundary, pml_layers=4)
        g.add_source(PlaneWave(frequency=2e9, y=7))
        g.add_conductor(Wall(y=20, gap_start=10, gap_end=18))
        g._prepare(g.default_dt(), 0.0, 2 * STEPS)
        return g

    def step(g):
        nat.check(lib.jxf_grid2d_step(g._h, STEPS, nat.stream_handle()), "step")

    def fields(g):
        out = np.empty((3,) + g.size, dtype=np.float32)
        for c in range(3):
            nat.check(lib.jxf_grid2d_get_field(g._h, c, out[c].ctypes.data, 1,
                                               nat.stream_handle()), "get")
        return out

    g, ref = grid(), grid()
    _capture_and_replay(lambda: step(g))
    step(ref)
    assert np.array_equal(fields(g), fields(ref))
    step(g)
    step(ref)
    assert np.array_equal(fields(g), fields(ref)) and np.abs(fields(g)).max() > 0
