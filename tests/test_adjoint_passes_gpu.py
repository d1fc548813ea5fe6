"""The transposed step's passes (``csrc/fdtd3d_adjoint.cuh``) against FP64
reverse-mode autodiff, at the shapes where their work split changes: odd and
even rows, slabs that cover a whole axis, several blocks per region with
remainders, stretched layers, sources in the slabs, E and H probes on faces
and repeated, and both ways of keeping the recomputed states (left by the E
pass, and copied after a TMA step).

Tolerance: a cell's adjoint goes through about ten FP32 operations a step, so
60 steps leave at most 60 * 10 * 6e-8 = 3.6e-5 of relative error; 1e-4.
"""

import numpy as np
import pytest

from cases import rn
from gpu_helpers import rel_l2, smooth_eps, to_np

pytestmark = pytest.mark.gpu

STEPS = 60


def _compare(cuda, size, layers, boundary, path, sources, probes, every=9):
    import torch

    from jaxphys_b200 import CPMLSpec, EMGrid3D, PointSource3D
    from jaxphys_b200.em.adjoint import probe_traces
    from oracle import torch_ref

    kw, spec_kw = {}, {}
    bnd = boundary
    if boundary == "stretched":
        bnd = "cpml"
        kw["cpml"] = CPMLSpec(kappa_max=4.0, alpha_max=0.03)
        spec_kw["cpml"] = rn.CpmlParams(kappa_max=4.0, alpha_max=0.03)
    dt = rn.default_dt_3d(1.0)
    eps = smooth_eps(size, 1.0, 4.0, seed=7)
    sources = [dict(frequency=f / dt, position=p, polarization=pol, waveform="gauss_sine",
                    width_steps=width, amplitude=amp) for f, p, pol, width, amp in sources]
    g = EMGrid3D(size=size, resolution=1.0, boundary=bnd, pml_layers=layers, path=path, **kw)
    for s in sources:
        g.add_source(PointSource3D(**s))
    for p in probes:
        g.add_probe(p[:3], ("ex", "ey", "ez", "hx", "hy", "hz")[p[3]])
    g.prepare(dt=dt)
    # H probes weighted to the size of the E ones (eta0)
    w = np.random.default_rng(1).random((STEPS, len(probes)))
    w[:, 3:] *= 377.0**2
    e = torch.tensor(eps, dtype=torch.float32, device=cuda, requires_grad=True)
    tr = probe_traces(g, e, STEPS, checkpoint_every=every)
    (torch.as_tensor(w, dtype=torch.float32, device=cuda) * tr**2).sum().backward()

    src64 = [dict(position=s["position"], polarization=s["polarization"],
                  amplitude=s.get("amplitude", 1.0), kind="gauss_sine", frequency=s["frequency"],
                  width_steps=s["width_steps"], delay_steps=4 * s["width_steps"])
             for s in sources]
    spec = rn.Spec3D(size=size, dx=1.0, boundary=bnd, pml_layers=layers, eps_r=eps, sources=src64,
                     probes=probes, **spec_kw)
    eps32 = eps.astype(np.float32).astype(np.float64)
    _, grad64, tr64 = torch_ref.grad_eps(spec, eps32, STEPS, dt, w)
    assert rel_l2(to_np(tr), tr64) <= 1e-5
    assert rel_l2(to_np(e.grad), grad64) <= 1e-4


@pytest.mark.parametrize("path", ["auto", "tma"])
@pytest.mark.parametrize("size,layers,boundary", [
    ((11, 9, 13), 2, "cpml"),
    ((12, 14, 10), 3, "stretched"),
    ((8, 15, 12), 6, "cpml"),
    ((14, 22, 52), 4, "stretched"),
    ((13, 40, 44), 5, "cpml"),
    ((10, 9, 16), 3, "pec"),
], ids=str)
def test_gradient_matches_fp64_autodiff(cuda, size, layers, boundary, path):
    nx, ny, nz = size
    if path == "tma" and nz % 4:
        pytest.skip("the TMA path needs nz % 4 == 0")
    sources = [(0.06, (nx // 2, ny // 2, nz // 2), "z", 5.0, 1.0), (0.05, (1, ny - 2, 1), "x", 4.0, 0.7)]
    probes = [(nx // 2, ny // 2, nz - 2, 2), (nx // 2, ny // 2, nz - 2, 2), (nx - 1, 2, 2, 1),
              (2, 0, nz // 2, 3), (nx // 3, ny - 2, 1, 5)]
    _compare(cuda, size, layers, boundary, path, sources, probes)


@pytest.mark.parametrize("size", [(13, 15, 17), (12, 17, 14)], ids=str)
def test_gradient_in_damping_layers(cuda, size):
    """Odd and even rows of a grid with damping layers; sources and probes
    between them (in the layers a field falls below FP32's range)."""
    nx, ny, nz = size
    c = (nx // 2, ny // 2, nz // 2)
    probes = [(*c, 0), (c[0] - 1, c[1], c[2] + 2, 2), (c[0] + 1, c[1] - 2, c[2], 4)]
    sources = [(0.06, c, "z", 5.0, 1.0), (0.05, (c[0], c[1] + 2, c[2] - 2), "x", 4.0, 0.7)]
    _compare(cuda, size, 3, "absorbing", "auto", sources, probes)


@pytest.mark.parametrize("keep", [None, "0", "25", "59"])
def test_kept_and_recomputed_steps(cuda, monkeypatch, keep):
    """Snapshots kept by the forward run for all, none, some and all but one
    of the steps."""
    if keep is not None:
        monkeypatch.setenv("JXF_ADJ_KEEP", keep)
    size = (12, 15, 14)
    sources = [(0.06, (6, 7, 7), "z", 5.0, 1.0), (0.05, (1, 13, 1), "x", 4.0, 0.7)]
    probes = [(6, 7, 12, 2), (11, 2, 2, 1), (2, 0, 7, 3)]
    _compare(cuda, size, 3, "cpml", "auto", sources, probes, every=None)


def test_step_counts_in_turn(cuda):
    """The buffer of kept snapshots is sized for the longest run so far: runs
    of other lengths on the same grid give what a new grid gives."""
    import torch

    from jaxphys_b200 import EMGrid3D, PointSource3D
    from jaxphys_b200.em.adjoint import probe_traces

    size = (12, 15, 14)
    eps = torch.tensor(smooth_eps(size, 1.0, 4.0, seed=7), dtype=torch.float32, device=cuda)

    def grid():
        g = EMGrid3D(size=size, resolution=1.0, boundary="cpml", pml_layers=3)
        g.add_source(PointSource3D(frequency=0.06 / rn.default_dt_3d(1.0), position=(6, 7, 7),
                                   waveform="gauss_sine", width_steps=5.0))
        g.add_probe((6, 7, 12), "ez")
        g.prepare(dt=rn.default_dt_3d(1.0))
        return g

    def grad(g, steps):
        e = eps.clone().requires_grad_(True)
        (probe_traces(g, e, steps) ** 2).sum().backward()
        return to_np(e.grad)

    used = grid()
    for steps in (30, 60, 1, 45, 60):
        got = grad(used, steps)
        assert np.array_equal(got, grad(grid(), steps)), steps
