"""Several 2D steps per launch (``k2d_steps``) against the one-step kernels
(which single-step calls run): equal values, no tolerance, over both window
shapes, launches of 1 to 10 steps, grids narrower than a window and with
ragged tiles, edge rules crossing windows, sources and walls on and next to
the edges, more sources than a block keeps samples of."""

import numpy as np
import pytest

from gpu_helpers import to_np

pytestmark = pytest.mark.gpu

SIZES = [(10, 10), (11, 57), (40, 33), (151, 203), (65, 300)]


def _grid(size, boundary, many):
    from jaxphys_b200 import EMGrid, PlaneWave, Wall

    nx, ny = size
    g = EMGrid(size=size, resolution=0.01, boundary=boundary, pml_layers=4)
    rows = [0, 1, ny // 2, ny // 2, ny - 2, ny - 1]
    for i, y in enumerate(rows * (4 if many else 1)):
        g.add_source(PlaneWave(frequency=(1.0 + 0.5 * (i % 3)) * 1e9, y=y, amplitude=0.5 + i))
    g.add_conductor(Wall(y=ny // 3, gap_start=nx // 4, gap_end=nx // 2))
    g.add_conductor(Wall(y=1, gap_start=2, gap_end=nx - 1))
    g.add_conductor(Wall(y=ny - 3))
    return g


def _single_steps(g, n):
    """Fields after each of n steps, one step per call."""
    from jaxphys_b200 import _native as nat

    import torch

    g._prepare(g.default_dt(), 0.0, n)
    lib, st = nat.load(), nat.stream_handle()
    out = torch.empty((3, n) + g.size, dtype=torch.float32, device="cuda")
    for k in range(n):
        nat.check(lib.jxf_grid2d_step(g._h, 1, st), "step")
        for c in range(3):
            nat.check(lib.jxf_grid2d_get_field(g._h, c, out[c, k].data_ptr(), 0, st), "get")
    return to_np(out)


@pytest.mark.parametrize("launch", [None, "0,1", "0,6", "0,10", "1,4", "1,9"])
@pytest.mark.parametrize("boundary", ["absorbing", "periodic", "reflecting"])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_steps_equal_single_steps(cuda, monkeypatch, size, boundary, launch):
    from jaxphys_b200 import _native as nat

    if launch is not None:
        monkeypatch.setenv("JXF_BLOCK2D", launch)
    n = 25
    many = launch == "0,6"
    want = _single_steps(_grid(size, boundary, many), n)
    assert np.abs(want).max() > 0
    g = _grid(size, boundary, many)
    span = (0.0, (n + 0.5) * g.default_dt())
    for every in (1, 7, 12):  # 25 steps end on a frame, after one, and between two
        h = g.simulate(t_span=span, save_every=every)
        for c, k in enumerate(("ez", "hx", "hy")):
            assert np.array_equal(to_np(getattr(h, k)), want[c, ::every]), (every, k)
    # the state after the run, and steps that go on from it in two calls
    g._prepare(g.default_dt(), 0.0, n)
    lib, st = nat.load(), nat.stream_handle()
    for part in (11, 14):
        nat.check(lib.jxf_grid2d_step(g._h, part, st), "step")
    for c in range(3):
        got = np.empty(size, dtype=np.float32)
        nat.check(lib.jxf_grid2d_get_field(g._h, c, got.ctypes.data, 1, st), "get")
        assert np.array_equal(got, want[c, -1]), c
