"""In-place two-pass steps (``csrc/fdtd3d_sweep.cuh``) against the per-cell
kernels that a generic batch of one grid runs (periodic grids, which are not
batched: against the FP32 oracle): equal values (the same roundings in the
same order, so no tolerance; only the sign of an exact zero may differ), over the shapes where the work split of a plane changes: every
vector width (nz % 4, nz % 2, odd nz), slabs that cover a whole axis, middles
narrower than a vector, blocks with remainders, stretched layers, sources on
faces, corners and region seams, duplicate sources, probes of all components.
"""

import numpy as np
import pytest

from cases import rn
from gpu_helpers import grid_fields, smooth_eps, to_np

pytestmark = pytest.mark.gpu

SHAPES = [
    # size, CPML layers (psi slabs are layers + 1 cells wide)
    ((9, 9, 8), 2),
    ((20, 21, 24), 3),    # 8-cell columns between the z regions
    ((21, 19, 22), 4),    # nz % 4 == 2
    ((18, 23, 27), 5),    # odd nz
    ((10, 33, 64), 6),    # slabs cover the whole x axis
    ((33, 12, 20), 7),    # ... and y and z
    ((24, 40, 132), 10),  # several blocks per region, remainders in each
]
FIELDS = ("ex", "ey", "ez", "hx", "hy", "hz")
BOUNDARIES = ["cpml", "stretched", "absorbing", "pec", "periodic"]


def _scene(size, layers):
    """Sources (frequency * dt, cell, amplitude, polarization) and probes; the
    amplitudes are powers of two, so scaling a sample rounds nothing."""
    nx, ny, nz = size
    p = layers + 1
    cells = [(nx // 2, ny // 2, nz // 2), (nx // 2, ny // 2, nz // 2), (0, 0, 0),
             (nx - 1, ny - 1, nz - 1), (1, min(p, ny - 1), min(p, nz - 1)),
             (nx // 2, max(ny - p, 0), max(nz - p, 0)), (nx // 2, ny - 1, 1)]
    sources = [(0.03 + 0.01 * (i % 3), c, 2.0 ** (i % 4), "xyz"[i % 3])
               for i, c in enumerate(cells)]
    sources.append((0.05, cells[0], 1.0, "x"))
    probes = [(c, k) for k in range(6)
              for c in ((nx // 2 - 1, ny // 2, nz // 2 + 1), (1, ny - 2, nz - 2))]
    return sources, probes


def _grid(size, layers, boundary, eps, path):
    from jaxphys_b200 import CPMLSpec, EMGrid3D, PointSource3D

    kw = {}
    if boundary == "stretched":
        kw["cpml"] = CPMLSpec(kappa_max=4.0, alpha_max=0.03)
        boundary = "cpml"
    g = EMGrid3D(size=size, resolution=1.0, boundary=boundary, pml_layers=layers, path=path, **kw)
    dt = g.default_dt()
    sources, probes = _scene(size, layers)
    for f, c, amp, pol in sources:
        g.add_source(PointSource3D(frequency=f / dt, position=c, amplitude=amp, polarization=pol))
    for c, k in probes:
        g.add_probe(c, FIELDS[k])
    if eps is not None:
        g.set_permittivity(eps)
    g.prepare(dt=dt)
    return g


def _reference(size, layers, boundary, eps, runs):
    """Traces of each run and the fields after the last one."""
    from jaxphys_b200.em.batch import FDTDBatch

    if boundary != "periodic":
        ref = _grid(size, layers, boundary, eps, "generic")
        batch = FDTDBatch([ref])
        assert batch.path == "generic"
        return [to_np(batch.run(n)[0]) for n in runs], grid_fields(ref)
    dt = rn.default_dt_3d(1.0)
    sources, probes = _scene(size, layers)
    o = rn.Oracle3D(rn.Spec3D(
        size=size, dx=1.0, boundary="periodic", eps_r=eps,
        sources=[dict(frequency=f / dt, position=c, amplitude=a, polarization=p)
                 for f, c, a, p in sources],
        probes=[(*c, k) for c, k in probes]), dt=dt, dtype=np.float32)
    return [o.run(n)["probes"].astype(np.float32) for n in runs], o.f


@pytest.mark.parametrize("with_eps", [False, True])
@pytest.mark.parametrize("boundary", BOUNDARIES)
@pytest.mark.parametrize("size,layers", SHAPES, ids=lambda v: str(v))
def test_sweep_equals_per_cell_kernels(cuda, size, layers, boundary, with_eps):
    eps = smooth_eps(size, 1.0, 6.0, seed=3) if with_eps else None
    runs = (7, 12)  # the second run starts where the first one ended
    want, fields = _reference(size, layers, boundary, eps, runs)
    g = _grid(size, layers, boundary, eps, "auto")
    got = [to_np(g.run(n)) for n in runs]
    g.check()
    assert g.kernels_per_step() == 2
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.abs(got[1]).max() > 0
    for name, a, b in zip(FIELDS, grid_fields(g), fields):
        assert np.array_equal(a, b), name
