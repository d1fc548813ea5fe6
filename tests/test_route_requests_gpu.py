"""Requests for a kernel path are honoured where in-place passes are the
default: calls that pin a TMA launch end the passes, and ``path="generic"``
runs the per-cell kernels.  Equal values on every route."""

import numpy as np
import pytest

from gpu_helpers import grid_fields, smooth_eps, to_np

pytestmark = pytest.mark.gpu

SIZE = (22, 20, 24)


def _grid(path, boundary="cpml", size=SIZE, eps=True):
    from jaxphys_b200 import EMGrid3D, PointSource3D

    g = EMGrid3D(size=size, resolution=1.0, boundary=boundary, pml_layers=4, path=path)
    g.add_source(PointSource3D(frequency=0.05 / g.default_dt(),
                               position=tuple(s // 2 for s in size)))
    for c in ("ez", "hx"):
        g.add_probe((size[0] // 2 + 1, size[1] // 2, size[2] // 2), c)
    if eps:
        g.set_permittivity(smooth_eps(size, 1.0, 4.0, seed=2))
    g.prepare()
    return g


@pytest.mark.parametrize("call", ["axis_split", "launch", "blocked"])
def test_pinned_launch_ends_the_passes(cuda, call):
    from jaxphys_b200 import _native as nat

    g = _grid("auto")
    traces = [to_np(g.run(7))]
    assert g.info()["tma_config"] == -1 and g.kernels_per_step() == 2
    lib = nat.load()
    rc = {"axis_split": lambda: lib.jxf_grid3d_set_axis_split(g._h, 1),
          "launch": lambda: lib.jxf_grid3d_set_launch(g._h, 0, 8),
          "blocked": lambda: lib.jxf_grid3d_set_blocked(g._h, 0, 8)}[call]()
    nat.check(rc, call)
    traces.append(to_np(g.run(8)))
    assert g.info()["tma_config"] >= 0
    ref = _grid("tma")
    assert np.array_equal(np.vstack(traces), to_np(ref.run(15)))
    for a, b in zip(grid_fields(g), grid_fields(ref)):
        assert np.array_equal(a, b)
