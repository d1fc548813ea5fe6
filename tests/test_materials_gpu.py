"""Materials uploaded as masks: the update factors they give equal those of
the per-cell permittivity array, on grids with and without a remainder of
four cells; frames written by the native run equal copies of the fields."""

import numpy as np
import pytest

from gpu_helpers import to_np

pytestmark = pytest.mark.gpu


def _grid(size, boundary):
    from jaxphys_b200 import EMGrid3D, PointSource3D

    g = EMGrid3D(size=size, boundary=boundary, pml_layers=3)
    g.add_source(PointSource3D(frequency=3e9, position=tuple(s // 2 for s in size)))
    return g


@pytest.mark.parametrize("conductor", [False, True])
@pytest.mark.parametrize("size", [(12, 11, 9), (10, 14, 16)])
def test_masks_equal_permittivity(cuda, size, conductor):
    from jaxphys_b200 import DielectricRegion

    rng = np.random.default_rng(2)
    m1, m2 = rng.random(size) < 0.4, (rng.random(size) < 0.2).astype(np.int32)
    metal = rng.random(size) < 0.1
    a, b = _grid(size, "absorbing"), _grid(size, "absorbing")
    a.add_material(DielectricRegion(mask=m1, epsilon_r=2.7))
    a.add_material(DielectricRegion(mask=np.asfortranarray(m2), epsilon_r=5))
    if conductor:
        a.add_conductor(metal)
        b.add_conductor(metal)
    eps = np.where(m2, 5.0, np.where(m1, 2.7, 1.0))
    b.set_permittivity(eps)
    span = (0.0, 30.5 * a.default_dt())
    for _ in range(2):  # the second run uploads the masks again
        u = a.simulate(t_span=span, save_every=7)
    v = b.simulate(t_span=span, save_every=7)
    host = b.simulate(t_span=span, save_every=7, history="host")
    for k in ("ex", "ey", "ez", "hx", "hy", "hz"):
        assert np.array_equal(to_np(getattr(u, k)), to_np(getattr(v, k))), k
        assert np.array_equal(to_np(getattr(v, k)), to_np(getattr(host, k))), k
    assert np.abs(to_np(u.ez)).max() > 0
