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


@pytest.mark.parametrize("boundary", ["cpml", "absorbing", "pec", "periodic"])
def test_generic_path_runs_the_per_cell_kernels(cuda, boundary):
    """Three launches a step (H, E, sources), whole grids of every boundary."""
    for size in (SIZE, (11, 14, 13)):
        g, ref = _grid("generic", boundary, size), _grid("auto", boundary, size)
        got = np.vstack([to_np(g.run(9)), to_np(g.run(6))])
        want = to_np(ref.run(15))
        assert g.kernels_per_step() == 3 and ref.kernels_per_step() == 2
        assert np.array_equal(got, want) and np.abs(want).max() > 0
        for a, b in zip(grid_fields(g), grid_fields(ref)):
            assert np.array_equal(a, b)


def test_gradient_of_a_generic_grid(cuda):
    """The adjoint of a per-cell grid recomputes with the same kernels."""
    import torch

    from jaxphys_b200.em.adjoint import probe_traces

    grads = []
    for path in ("generic", "auto"):
        g = _grid(path, "cpml", (12, 13, 14), eps=False)
        e = torch.tensor(smooth_eps((12, 13, 14), 1.0, 4.0, seed=5), dtype=torch.float32,
                         device=cuda, requires_grad=True)
        (probe_traces(g, e, 30) ** 2).sum().backward()
        grads.append(to_np(e.grad))
        assert g.kernels_per_step() == (3 if path == "generic" else 2)
    assert np.array_equal(grads[0], grads[1]) and np.abs(grads[0]).max() > 0
