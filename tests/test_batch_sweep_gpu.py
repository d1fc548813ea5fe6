"""Batches on in-place sweeps (one group of grids after the other, several
grids per launch) against every grid stepped alone: equal values, no
tolerance.  More grids than a launch holds, mixed vector widths, grids with
and without permittivity maps where the per-grid kernels allow it, probes of
E and H, two runs in a row, and the learned band."""

import numpy as np
import pytest

from gpu_helpers import smooth_eps, to_np

pytestmark = pytest.mark.gpu

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")
EVEN = [(20, 24, 28), (33, 21, 16), (12, 40, 32), (24, 24, 24), (17, 16, 20), (30, 12, 36),
        (18, 18, 16), (22, 26, 24), (14, 14, 12), (28, 20, 40), (9, 11, 12)]
MIXED = [(20, 24, 27), (18, 22, 26), (21, 19, 24), (16, 30, 33)]


def _grid(i, size, boundary, path, eps=True):
    from jaxphys_b200 import EMGrid3D, PointSource3D

    g = EMGrid3D(size=size, resolution=1.0, boundary=boundary, pml_layers=4, path=path)
    dt = g.default_dt()
    c = tuple(s // 2 for s in size)
    for k, pos in enumerate((c, (0, size[1] - 1, 3), c)):
        g.add_source(PointSource3D(frequency=(0.04 + 0.01 * k) / dt, position=pos,
                                   polarization="xyz"[(i + k) % 3], amplitude=1.0 + k))
    if i % 3 != 2:
        g.add_probe((c[0], c[1], min(c[2] + 3, size[2] - 1)), "ez")
        g.add_probe((1, 2, 3), "hx")
    if i % 4 == 1:  # an outermost cell, which a band corrects after the E pass
        g.add_probe((0, 2, 3), "hy")
    if eps:
        g.set_permittivity(smooth_eps(size, 1.0, 3.0 + i % 4, seed=i))
    g.prepare(dt=dt)
    return g


@pytest.mark.parametrize("boundary", ["cpml", "absorbing", "pec"])
@pytest.mark.parametrize("sizes,eps", [(EVEN, True), (EVEN, False), (MIXED[:2], True),
                                       (MIXED[::3], False)])
def test_sweep_batch_equals_grids_alone(cuda, monkeypatch, boundary, sizes, eps):
    from jaxphys_b200.em.batch import FDTDBatch

    monkeypatch.setenv("JXF_BATCH_LAUNCH", "sweep")
    grids = [_grid(i, s, boundary, "auto", eps) for i, s in enumerate(sizes)]
    b = FDTDBatch(grids)
    first, second = b.run(9), b.run(14, use_graph=False)
    assert b.launch()["tma_config"] == -1 and b.kernels_per_step() % 2 == 0
    for i, s in enumerate(sizes):
        ref = _grid(i, s, boundary, "generic", eps)
        want = ref.run(23)
        if want is None:
            assert first[i] is None and second[i] is None
        else:
            assert np.array_equal(np.vstack([to_np(first[i]), to_np(second[i])]), to_np(want)), i
        for k in COMPS:
            assert np.array_equal(to_np(grids[i].field(k)), to_np(ref.field(k))), (i, k)
    b.reset()
    again = b.run(9)
    assert all(np.array_equal(to_np(u), to_np(v)) for u, v in zip(again, first) if u is not None)
    b.close()


def test_sweep_batch_learned_band_equals_lockstep(cuda, monkeypatch):
    from jaxphys_b200.em.batch import FDTDBatch
    from jaxphys_b200.em.learned import default_band

    sizes = EVEN[:10]
    out = {}
    for launch, path in (("sweep", "auto"), ("", "generic")):
        monkeypatch.setenv("JXF_BATCH_LAUNCH", launch)
        grids = [_grid(i, s, "pec", path) for i, s in enumerate(sizes)]
        b = FDTDBatch(grids)
        b.set_band(default_band())
        traces = b.run(13)
        out[path] = ([None if t is None else to_np(t) for t in traces],
                     [[to_np(g.field(k)) for k in COMPS] for g in grids])
        b.set_band(None)  # a detached band leaves the batch usable
        b.run(2)
        b.close()
    for u, v in zip(out["auto"][0], out["generic"][0]):
        assert (u is None) == (v is None) and (u is None or np.array_equal(u, v))
    for i in range(len(sizes)):
        for k in range(6):
            assert np.array_equal(out["auto"][1][i][k], out["generic"][1][i][k]), (i, k)
