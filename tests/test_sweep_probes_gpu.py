"""Probes recorded by the in-place passes: counts around a block's threads and
above a grid's, cells and components repeated, against the per-cell kernels
of a generic batch of one grid (equal values); and that many probes do not
serialise a step."""

import time

import numpy as np
import pytest

from gpu_helpers import to_np

pytestmark = pytest.mark.gpu

FIELDS = ("ex", "ey", "ez", "hx", "hy", "hz")


def _grid(size, boundary, probes, path):
    from jaxphys_b200 import EMGrid3D, PointSource3D

    rng = np.random.default_rng(probes)
    g = EMGrid3D(size=size, resolution=1.0, boundary=boundary, pml_layers=2, path=path)
    g.add_source(PointSource3D(frequency=0.05 / g.default_dt(),
                               position=tuple(s // 2 for s in size)))
    for _ in range(probes):
        g.add_probe(tuple(int(rng.integers(0, s)) for s in size), FIELDS[rng.integers(0, 6)])
    g.prepare()
    return g


@pytest.mark.parametrize("probes", [1, 127, 128, 129, 257, 4500])
@pytest.mark.parametrize("size,boundary", [((9, 9, 8), "cpml"), ((8, 10, 9), "absorbing")])
def test_probe_counts(cuda, size, boundary, probes):
    from jaxphys_b200.em.batch import FDTDBatch

    g = _grid(size, boundary, probes, "auto")
    got = np.vstack([to_np(g.run(7)), to_np(g.run(1)), to_np(g.run(5))])
    assert g.kernels_per_step() == 2
    b = FDTDBatch([_grid(size, boundary, probes, "generic")])
    want = to_np(b.run(13)[0])
    assert np.array_equal(got, want)
    assert probes == 1 or np.abs(want).max() > 0  # (the one probe reads no signal)
    b.close()


@pytest.mark.parametrize("batched", [False, True])
def test_many_probes_do_not_serialise_a_step(cuda, batched):
    """16,384 probes are a block's width times 128: recorded by one block they
    cost 24 steps, spread over the blocks a fraction of one."""
    import torch

    from jaxphys_b200.em.batch import FDTDBatch

    def us(probes):
        g = _grid((33, 33, 33), "cpml", probes, "auto")
        run = FDTDBatch([g]).run if batched else g.run
        run(64)
        best = 1e9
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            run(64)
            torch.cuda.synchronize()
            best = min(best, (time.perf_counter() - t0) / 64 * 1e6)
        return best

    assert us(16384) < 4.0 * us(1)
