"""What a batch with nz % 4 != 0 runs: lockstep launches for the whole batch
where its groups would be many and small, groups of in-place passes where
they are faster; equal values either way."""

import numpy as np
import pytest

from gpu_helpers import to_np

pytestmark = pytest.mark.gpu

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")


def _run(n, side, boundary, path, steps=6, band=False):
    from jaxphys_b200 import EMGrid3D, PointSource3D
    from jaxphys_b200.em.batch import FDTDBatch
    from jaxphys_b200.em.learned import default_band

    grids = []
    for i in range(n):
        g = EMGrid3D(size=(side, side, side), resolution=1.0, boundary=boundary, pml_layers=4,
                     path=path)
        g.add_source(PointSource3D(frequency=0.05 / g.default_dt(), polarization="xyz"[i % 3],
                                   position=(side // 2,) * 3))
        g.add_probe((side // 2 + 1,) * 3, "ez")
        g.prepare()
        grids.append(g)
    b = FDTDBatch(grids)
    if band:
        b.set_band(default_band())
    traces = [to_np(t) for t in b.run(steps)]
    fields = [[to_np(g.field(k)) for k in COMPS] for g in grids]
    launches = b.kernels_per_step()
    b.close()
    return traces, fields, launches


@pytest.mark.parametrize("n,side,boundary,band,launches", [
    (64, 17, "pec", False, 4),     # lockstep: H, E, sources, probes
    (64, 17, "cpml", False, 4),
    (64, 17, "pec", True, 6),      # ... and two for the band
    (200, 9, "absorbing", False, 4),
    (8, 17, "pec", False, 2),      # one group
    (16, 33, "cpml", False, 4),    # two groups
    (8, 17, "pec", True, 4),
])
def test_launches_of_small_batches(cuda, n, side, boundary, band, launches):
    traces, fields, got = _run(n, side, boundary, "auto", band=band)
    assert got == launches
    want_traces, want_fields, _ = _run(n, side, boundary, "generic", band=band)
    for i in range(n):
        assert np.array_equal(traces[i], want_traces[i]), i
        for k in range(6):
            assert np.array_equal(fields[i][k], want_fields[i][k]), (i, k)


def test_band_weighs_in_the_choice(cuda):
    """A band attached after a run makes the batch choose again; the state
    goes on from where it was."""
    from jaxphys_b200 import EMGrid3D
    from jaxphys_b200.em.batch import FDTDBatch
    from jaxphys_b200.em.learned import default_band

    out = {}
    for path in ("auto", "generic"):
        # 16 grids of 57^3: groups without a band, lockstep with one
        grids = [EMGrid3D(size=(57, 57, 57), resolution=1.0, boundary="pec", path=path)
                 for _ in range(16)]
        for i, g in enumerate(grids):
            g.prepare()
            g.set_field("ez", np.random.default_rng(i).standard_normal(g.size).astype(np.float32))
        b = FDTDBatch(grids)
        b.run(3)
        launches = [b.kernels_per_step()]
        b.set_band(default_band())
        b.run(3)
        launches.append(b.kernels_per_step())
        b.set_band(None)
        b.run(3)
        launches.append(b.kernels_per_step())
        out[path] = launches, [to_np(g.field(k)) for g in grids for k in COMPS]
        b.close()
    assert out["generic"][0] == [2, 4, 2]
    assert out["auto"][0] == [4, 4, 4]  # (two groups; lockstep with a band; two groups)
    for u, v in zip(out["auto"][1], out["generic"][1]):
        assert np.array_equal(u, v)
