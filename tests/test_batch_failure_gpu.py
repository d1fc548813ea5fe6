"""Batches on in-place passes whose first run meets a refused device
allocation (``JXF_FAULT_ALLOC_AFTER``): the call raises, no grid has stepped,
and a later call gives what a batch that never failed gives.  And a batch that tries
the passes but keeps lockstep holds one set of band tables."""

import numpy as np
import pytest

from gpu_helpers import to_np

pytestmark = pytest.mark.gpu

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")
# more grids than one group holds
SIZES = [(20, 24, 28), (33, 21, 16), (12, 40, 32), (24, 24, 24), (17, 16, 20), (30, 12, 36),
         (18, 18, 16), (22, 26, 24), (14, 14, 12), (28, 20, 40)]


def _batch(sources=False):
    from jaxphys_b200 import EMGrid3D, PointSource3D
    from jaxphys_b200.em.batch import FDTDBatch

    grids = []
    for i, size in enumerate(SIZES):
        g = EMGrid3D(size=size, resolution=1.0, boundary="pec")
        if sources:
            g.add_source(PointSource3D(frequency=0.05 / g.default_dt(), position=(3, 4, 5)))
        g.prepare()
        g.set_field("ez", np.random.default_rng(i).standard_normal(size).astype(np.float32))
        g.add_probe(tuple(s // 2 for s in size), "ey")
        grids.append(g)
    return grids, FDTDBatch(grids)


def _fields(grids):
    return [to_np(g.field(k)) for g in grids for k in COMPS]


def _run_past_refusals(monkeypatch, grids, batch, steps):
    """Run with 0, 1, 2, ... allocations allowed until one call succeeds."""
    from jaxphys_b200 import SimulationError

    before = _fields(grids)
    for n in range(300):
        monkeypatch.setenv("JXF_FAULT_ALLOC_AFTER", str(n))
        try:
            out = batch.run(steps)
        except SimulationError as e:
            assert "fault injection" in str(e)
        else:
            monkeypatch.delenv("JXF_FAULT_ALLOC_AFTER")
            return n, out
        monkeypatch.delenv("JXF_FAULT_ALLOC_AFTER")
        for a, b in zip(_fields(grids), before):
            assert np.array_equal(a, b), n
    raise AssertionError("the run never succeeded")


def test_refused_band_tables(cuda, monkeypatch):
    """Every group keeps its band: none steps as bare PEC after a refusal."""
    from jaxphys_b200.em.learned import default_band

    monkeypatch.setenv("JXF_BATCH_LAUNCH", "sweep")
    grids, batch = _batch()
    batch.set_band(default_band())
    refused, got = _run_past_refusals(monkeypatch, grids, batch, 9)
    assert refused > 5  # the tables of both groups
    ref_grids, ref = _batch()
    ref.set_band(default_band())
    want = ref.run(9)
    for a, b in zip(got, want):
        assert np.array_equal(to_np(a), to_np(b))
    for a, b in zip(_fields(grids), _fields(ref_grids)):
        assert np.array_equal(a, b)
    batch.close()
    ref.close()


def test_refused_source_lists(cuda, monkeypatch):
    """No group has stepped when the source lists of a later one are refused."""
    monkeypatch.setenv("JXF_BATCH_LAUNCH", "sweep")
    grids, batch = _batch(sources=True)
    refused, got = _run_past_refusals(monkeypatch, grids, batch, 9)
    # (finished lists are kept, so each call gets further: the last ones into
    # the second group)
    assert refused >= 8
    ref_grids, ref = _batch(sources=True)
    want = ref.run(9)
    for a, b in zip(got, want):
        assert np.array_equal(to_np(a), to_np(b))
    for a, b in zip(_fields(grids), _fields(ref_grids)):
        assert np.array_equal(a, b)
    batch.close()
    ref.close()


@pytest.mark.parametrize("launch", ["sweep", "0,8"])
def test_refused_longer_probe_buffer(cuda, monkeypatch, launch):
    """A refused buffer for a longer run does not cost the shorter runs after
    it their probe rows."""
    from jaxphys_b200 import SimulationError

    monkeypatch.setenv("JXF_BATCH_LAUNCH", launch)
    grids, batch = _batch(sources=True)
    first = batch.run(4)
    monkeypatch.setenv("JXF_FAULT_ALLOC_AFTER", "0")
    with pytest.raises(SimulationError, match="fault injection"):
        batch.run(9)
    monkeypatch.delenv("JXF_FAULT_ALLOC_AFTER")
    second = batch.run(3)
    ref_grids, ref = _batch(sources=True)
    want = ref.run(7)
    for a, b, c in zip(first, second, want):
        assert np.array_equal(np.vstack([to_np(a), to_np(b)]), to_np(c))
    batch.close()
    ref.close()


def test_lockstep_holds_one_set_of_band_tables(cuda, monkeypatch):
    """Two batches in turn on grids above the L2, where lockstep is faster:
    one tunes (and so tries the passes), one is pinned to the shape found.  A
    second set of band tables would be 32 bytes for each of the outer cells."""
    import gc

    import torch

    from jaxphys_b200 import EMGrid3D
    from jaxphys_b200.em.batch import FDTDBatch
    from jaxphys_b200.em.learned import default_band

    grids = [EMGrid3D(size=(256, 256, 256), resolution=1.0, boundary="pec") for _ in range(3)]
    for g in grids:
        g.prepare()
    band = default_band()
    second = 3 * 32 * (256**3 - 254**3)

    def used():
        gc.collect()
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info(0)
        return total - free

    taken = []
    for _ in range(2):
        batch = FDTDBatch(grids)
        batch.set_band(band)
        before = used()
        batch.run(2, use_graph=False)
        taken.append(used() - before)
        shape = batch.launch()
        if len(taken) == 1 and shape["tma_config"] < 0:
            pytest.skip("the passes were faster here")
        monkeypatch.setenv("JXF_BATCH_LAUNCH",
                           f"{shape['tma_config']},{shape['x_chunk']},{shape['axis_split']}")
        batch.close()
        batch = None
    assert taken[0] - taken[1] < second / 2, (taken, second)
