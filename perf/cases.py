"""Performance cases of the FDTD engine: what its users have it do.

Five kinds of work, each through the public entry points:

* ``grid2d``: ``EMGrid.simulate`` (2D TM, the reference's own call),
* ``grid3d``: ``EMGrid3D.simulate`` (3D, the reference's own call),
* ``run3d``:  ``EMGrid3D.reset`` / ``run`` with probes, then the fields (long
  CPML runs of one prepared grid),
* ``adjoint``: ``probe_traces`` forward and backward (inverse design),
* ``batch``:  ``FDTDBatch.run`` over many uneven grids.

``exact`` restates each in plain torch, FP64.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

from jaxphys_b200 import CPMLSpec, DielectricRegion, EMGrid, EMGrid3D, PlaneWave, PointSource3D, Wall
from jaxphys_b200.em.adjoint import probe_traces
from jaxphys_b200.em.batch import FDTDBatch

C0 = 299792458.0
MU0 = 4.0e-7 * math.pi
EPS0 = 1.0 / (MU0 * C0**2)
FIELDS3D = ("ex", "ey", "ez", "hx", "hy", "hz")
FIELDS2D = ("ez", "hx", "hy")
POL = {"x": 0, "y": 1, "z": 2}


# ------------------------------------------------------------------ the cases


def listed():
    return [
        # the 2D solver's documented example: one slit, every default
        dict(name="2d_slit_200", kind="grid2d", nx=200, ny=200, boundary="absorbing", walls=1,
             steps=428, save_every=10),
        # a small closed 2D box, odd sides, mirrored edges
        dict(name="2d_mirror_151x203", kind="grid2d", nx=151, ny=203, boundary="reflecting",
             walls=1, steps=300, save_every=10),
        # a large 2D diffraction scene
        dict(name="2d_slit_1024", kind="grid2d", nx=1024, ny=1024, boundary="absorbing", walls=2,
             steps=500, save_every=25),
        # the 3D solver with every default: size, layers, span, saved frames
        dict(name="3d_default_60", kind="grid3d", nx=60, ny=60, nz=60, boundary="absorbing",
             layers=8, materials=0, steps=262, save_every=20),
        # a periodic cell with dielectric inclusions (band structures, gratings)
        dict(name="3d_periodic_96x80x64", kind="grid3d", nx=96, ny=80, nz=64, boundary="periodic",
             layers=8, materials=2, steps=300, save_every=50),
        # a small antenna box with CPML walls, 500 steps
        dict(name="3d_cpml_64", kind="run3d", nx=64, ny=64, nz=64, boundary="cpml", layers=8,
             eps="vacuum", stretched=False, steps=500, probes=8),
        # the headline: 128^3, 1000 steps, dielectric sphere, 10-cell CPML
        dict(name="3d_cpml_128", kind="run3d", nx=128, ny=128, nz=128, boundary="cpml", layers=10,
             eps="sphere", stretched=False, steps=1000, probes=16),
        # odd sides, and the stretched (kappa > 1, CFS alpha) layers of waveguide work
        dict(name="3d_cpml_odd_75x90x61", kind="run3d", nx=75, ny=90, nz=61, boundary="cpml",
             layers=10, eps="smooth", stretched=True, steps=300, probes=4),
        # the largest single grid: 512^3 in a graded dielectric
        dict(name="3d_cpml_512", kind="run3d", nx=512, ny=512, nz=512, boundary="cpml", layers=12,
             eps="smooth", stretched=False, steps=200, probes=16),
        # one gradient of an inverse design: plane source, 32^3 design cells
        dict(name="adjoint_96", kind="adjoint", n=96, boundary="cpml", layers=10, design=32,
             steps=2000),
        # 64 design candidates of mixed sizes advanced together, CPML walls
        dict(name="batch64_cpml", kind="batch", grids=64, lo=48, hi=160, layers=10,
             boundary="cpml", steps=50),
        # the same candidates behind the learned absorbing band
        dict(name="batch64_learned", kind="batch", grids=64, lo=48, hi=160, layers=3,
             boundary="learned", steps=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid2d", "grid2d", "grid3d", "grid3d", "run3d", "run3d", "adjoint", "batch"])
    if kind == "grid2d":
        steps = _log_int(rng, 40, 500)
        return dict(kind=kind, nx=_log_int(rng, 40, 1400), ny=_log_int(rng, 40, 1400),
                    boundary=rng.choice(["absorbing", "absorbing", "reflecting", "periodic"]),
                    walls=rng.randint(0, 2), steps=steps,
                    save_every=rng.choice([s for s in (5, 10, 20, 25, 50) if s >= steps / 50]))
    if kind == "grid3d":
        steps = _log_int(rng, 40, 300)
        return dict(kind=kind, nx=_log_int(rng, 16, 160), ny=_log_int(rng, 16, 160),
                    nz=_log_int(rng, 16, 160),
                    boundary=rng.choice(["absorbing", "absorbing", "periodic", "pec"]),
                    layers=rng.randint(4, 10), materials=rng.randint(0, 2), steps=steps,
                    save_every=rng.choice([s for s in (10, 20, 50) if s >= steps / 20]))
    if kind == "run3d":
        return dict(kind=kind, nx=_log_int(rng, 32, 256), ny=_log_int(rng, 32, 256),
                    nz=_log_int(rng, 32, 256), boundary="cpml", layers=rng.randint(6, 12),
                    eps=rng.choice(["vacuum", "sphere", "smooth"]),
                    stretched=rng.random() < 0.3, steps=_log_int(rng, 50, 500),
                    probes=rng.randint(1, 16))
    if kind == "adjoint":
        n = _log_int(rng, 28, 96)
        return dict(kind=kind, n=n, boundary=rng.choice(["cpml", "cpml", "absorbing"]), layers=8,
                    design=max(4, n // 3), steps=_log_int(rng, 50, 600))
    lo = rng.randint(28, 60)
    return dict(kind=kind, grids=_log_int(rng, 4, 24), lo=lo, hi=lo + rng.randint(8, 50),
                layers=10, boundary=rng.choice(["cpml", "cpml", "learned"]),
                steps=rng.randint(20, 50))


# ------------------------------------------------------------------ the inputs


def _smooth(shape, lo, hi, seed):
    """A smooth random map in [lo, hi]: coarse noise, trilinear (on the GPU)."""
    g = torch.Generator().manual_seed(int(seed))
    coarse = [max(2, s // 12) for s in shape]
    u = torch.rand([1, 1] + coarse, generator=g).cuda()
    u = torch.nn.functional.interpolate(u, size=tuple(shape), mode="trilinear",
                                        align_corners=True)[0, 0]
    return (lo + (hi - lo) * u).contiguous()


def _spec2d(case, seed):
    """Sources (frequency, y, amplitude) and walls (y, gap) of a 2D scene."""
    rng = random.Random(seed)
    nx, ny = case["nx"], case["ny"]
    sources = [(rng.uniform(1.0e9, 4.0e9), ny // 10 + rng.randint(0, ny // 12),
                rng.uniform(0.5, 2.0))]
    walls = []
    for k in range(case["walls"]):
        centre = nx // 2 + rng.randint(-(nx // 8), nx // 8)
        half = max(2, nx // 20)
        walls.append((ny * (k + 2) // 4, centre - half, centre + half))
    return sources, walls


def _spec3d(case, seed):
    """Sources (frequency, position, amplitude, polarization) and dielectric
    boxes (corners, eps_r) of a 3D scene."""
    rng = random.Random(seed)
    size = (case["nx"], case["ny"], case["nz"])
    # two crossed dipoles: every field component is driven
    sources = [(rng.uniform(1.0e9, 4.0e9), tuple(n // 2 + rng.randint(-(n // 8), n // 8) for n in size),
                rng.uniform(0.5, 2.0), pol) for pol in rng.sample("xyz", 2)]
    boxes = []
    for _ in range(case["materials"]):
        a = tuple(rng.randint(n // 8, n // 2) for n in size)
        boxes.append((a, tuple(p + max(2, n // 4) for p, n in zip(a, size)), rng.uniform(1.5, 6.0)))
    return sources, boxes


def _mask(size, a, b):
    m = np.zeros(size, dtype=bool)
    m[a[0]:b[0], a[1]:b[1], a[2]:b[2]] = True
    return m


def _dt(dx, dims):
    return float(0.99 * dx / (C0 * float(np.sqrt(float(dims)))))


def _spec_run(case, seed):
    """A pulsed and two continuous dipoles (crossed, so that every component
    is driven to the end), probes near them, permittivity map (None: vacuum)."""
    rng = random.Random(seed)
    size = (case["nx"], case["ny"], case["nz"])
    dt = _dt(1.0, 3)
    pos = tuple(n // 2 + rng.randint(-(n // 10), n // 10) for n in size)
    pols = rng.sample("xyz", 2)
    sources = [dict(frequency=rng.uniform(0.04, 0.06) / dt, position=pos,
                    amplitude=rng.uniform(0.5, 2.0), polarization=pols[0], width=20.0)]
    for pol in pols:
        at = tuple(n // 2 + rng.randint(-(n // 10), n // 10) for n in size)
        sources.append(dict(frequency=rng.uniform(0.02, 0.04) / dt, position=at,
                            amplitude=rng.uniform(0.1, 0.3), polarization=pol, width=None))
    probes = [(tuple(min(max(p + rng.randint(-n // 5, n // 5), 1), n - 2) for p, n in zip(pos, size)),
               rng.choice(FIELDS3D)) for _ in range(case["probes"])]
    if case["eps"] == "vacuum":
        eps = None
    elif case["eps"] == "smooth":
        eps = _smooth(size, 1.0, 12.0, seed)
    else:
        c = [n // 2 + rng.randint(-(n // 8), n // 8) for n in size]
        ax = [torch.arange(n, device="cuda", dtype=torch.float32) - m for n, m in zip(size, c)]
        r2 = ax[0][:, None, None]**2 + ax[1][None, :, None]**2 + ax[2][None, None, :]**2
        eps = torch.where(r2 <= float(min(size) // 6)**2, 4.0, 1.0).contiguous()
    return sources, probes, eps


def _spec_batch(case, seed):
    """(size, eps_r, source) of every grid; the sizes do not depend on the seed."""
    sizes = random.Random(5)
    rng = random.Random(seed)
    pad = 2 * case["layers"]
    dt = _dt(1.0, 3)
    out = []
    for k in range(case["grids"]):
        if sizes.random() < 0.5:
            size = (sizes.randint(case["lo"], case["hi"]),) * 3
        else:
            size = tuple(sizes.randint(case["lo"], case["hi"]) for _ in range(3))
        size = tuple(n + pad for n in size)
        size = (size[0], size[1], -(-size[2] // 4) * 4)  # padded for the persistent batch kernel
        pos = tuple(rng.randint(n // 3, n - n // 3) for n in size)
        out.append((size, _smooth(size, 1.0, 6.0, seed * 1000 + k),
                    dict(frequency=0.05 / dt, position=pos, amplitude=rng.uniform(0.5, 2.0),
                         polarization=rng.choice("xyz"), width=12.0)))
    return out


def _spec_adjoint(case, seed):
    """Plane Ex source, Ez probe, eps_r = 1 + 11 sigmoid(theta) in the middle."""
    rng = random.Random(seed)
    n, d = case["n"], case["design"]
    g = torch.Generator().manual_seed(int(seed))
    theta = torch.randn((d, d, d), generator=g).cuda()
    eps = torch.ones((n, n, n), device="cuda")
    a = (n - d) // 2
    eps[a:a + d, a:a + d, a:a + d] = 1.0 + 11.0 * torch.sigmoid(theta)
    dt = _dt(1.0, 3)
    width = 30.0 if case["steps"] >= 300 else case["steps"] / 10.0
    source = dict(frequency=0.05 / dt, z=max(n // 6 - 1, 9), amplitude=rng.uniform(0.5, 1.5),
                  width=width)
    probe = (n // 2 + rng.randint(-2, 2), n // 2 + rng.randint(-2, 2), n - max(n // 6, 10))
    return eps, source, probe


def _point(s):
    if s["width"] is None:  # continuous
        return PointSource3D(frequency=s["frequency"], position=s["position"],
                             amplitude=s["amplitude"], polarization=s["polarization"])
    return PointSource3D(frequency=s["frequency"], position=s["position"], amplitude=s["amplitude"],
                         polarization=s["polarization"], waveform="gauss_sine",
                         width_steps=s["width"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid2d":
        sources, walls = _spec2d(case, seed)
        g = EMGrid(size=(case["nx"], case["ny"]), boundary=case["boundary"])
        for f, y, amp in sources:
            g.add_source(PlaneWave(frequency=f, y=y, amplitude=amp))
        for y, g0, g1 in walls:
            g.add_conductor(Wall(y=y, gap_start=g0, gap_end=g1))
        span = (0.0, (case["steps"] + 0.5) * g.default_dt())
        return dict(kind=kind, grid=g, span=span, save_every=case["save_every"])
    if kind == "grid3d":
        sources, boxes = _spec3d(case, seed)
        size = (case["nx"], case["ny"], case["nz"])
        g = EMGrid3D(size=size, boundary=case["boundary"], pml_layers=case["layers"])
        for f, pos, amp, pol in sources:
            g.add_source(PointSource3D(frequency=f, position=pos, amplitude=amp, polarization=pol))
        for a, b, eps in boxes:
            g.add_material(DielectricRegion(mask=_mask(size, a, b), epsilon_r=eps))
        span = (0.0, (case["steps"] + 0.5) * g.default_dt())
        return dict(kind=kind, grid=g, span=span, save_every=case["save_every"])
    if kind == "run3d":
        sources, probes, eps = _spec_run(case, seed)
        cpml = CPMLSpec(kappa_max=5.0, alpha_max=0.02) if case["stretched"] else CPMLSpec()
        g = EMGrid3D(size=(case["nx"], case["ny"], case["nz"]), resolution=1.0, boundary="cpml",
                     pml_layers=case["layers"], cpml=cpml)
        for s in sources:
            g.add_source(_point(s))
        for pos, comp in probes:
            g.add_probe(pos, comp)
        if eps is not None:
            g.set_permittivity(eps)
        g.prepare()
        return dict(kind=kind, grid=g, steps=case["steps"])
    if kind == "adjoint":
        eps, source, probe = _spec_adjoint(case, seed)
        n = case["n"]
        g = EMGrid3D(size=(n, n, n), resolution=1.0, boundary=case["boundary"],
                     pml_layers=case["layers"])
        for i in range(n):
            for j in range(n):
                g.add_source(_point(dict(source, position=(i, j, source["z"]), polarization="x")))
        g.add_probe(probe, "ez")
        g.add_probe(probe, "ex")
        g.prepare()
        return dict(kind=kind, grid=g, eps=eps.requires_grad_(True), steps=case["steps"])
    grids = []
    for size, eps, source in _spec_batch(case, seed):
        g = EMGrid3D(size=size, resolution=1.0, boundary=case["boundary"],
                     pml_layers=case["layers"])
        g.add_source(_point(source))
        g.add_probe(tuple(p + 3 for p in source["position"]), "ez")
        g.set_permittivity(eps)
        g.prepare()
        grids.append(g)
    return dict(kind=kind, batch=FDTDBatch(grids), steps=case["steps"])


# ------------------------------------------------------------------ one pass


def run(state):
    kind = state["kind"]
    if kind in ("grid2d", "grid3d"):
        h = state["grid"].simulate(t_span=state["span"], save_every=state["save_every"])
        return {k: getattr(h, k) for k in (FIELDS2D if kind == "grid2d" else FIELDS3D)}
    if kind == "run3d":
        g = state["grid"]
        g.reset()
        traces = g.run(state["steps"])
        return {"traces": traces, **g.fields}
    if kind == "adjoint":
        traces = probe_traces(state["grid"], state["eps"], state["steps"])
        (grad,) = torch.autograd.grad((traces**2).sum(), state["eps"])
        return {"traces": traces.detach(), "grad": grad}
    b = state["batch"]
    b.reset()
    traces = b.run(state["steps"])
    out = {k: torch.cat([g.field(k).reshape(-1) for g in b.grids]) for k in FIELDS3D}
    return {"traces": torch.cat([t.reshape(-1) for t in traces]), **out}


def _psi_cells(size, layers):
    """Cells of the psi arrays over all three axes (4 arrays per axis)."""
    cells = 0
    for ax in range(3):
        n = size[ax]
        other = size[(ax + 1) % 3] * size[(ax + 2) % 3]
        cells += 4 * min(n, 2 * (layers + 1)) * other
    return cells


def work(case):
    """Bytes the path cannot do without: what a pass is given, read once, and
    what it returns, written once; and the update arithmetic of every step."""
    kind, steps = case["kind"], case["steps"]
    if kind == "grid2d":
        cells = case["nx"] * case["ny"]
        frames = -(-steps // case["save_every"])
        return {"bytes": 12 * cells * frames, "flops": 13 * cells * steps}
    if kind == "grid3d":
        cells = case["nx"] * case["ny"] * case["nz"]
        frames = -(-steps // case["save_every"])
        return {"bytes": 24 * cells * frames, "flops": 36 * cells * steps}
    if kind == "run3d":
        size = (case["nx"], case["ny"], case["nz"])
        cells = size[0] * size[1] * size[2]
        return {"bytes": cells * (24 + (0 if case["eps"] == "vacuum" else 4)),
                "flops": (36 * cells + 5 * _psi_cells(size, case["layers"])) * steps}
    if kind == "adjoint":
        size = (case["n"],) * 3
        cells = case["n"]**3
        psi = _psi_cells(size, case["layers"]) if case["boundary"] == "cpml" else 0
        # the forward steps, and the transposed steps with dJ/dcb
        return {"bytes": 8 * cells, "flops": ((36 + 36 + 12) * cells + 10 * psi) * steps}
    sizes = _batch_sizes(case)
    cells = sum(a * b * c for a, b, c in sizes)
    extra = 0
    for s in sizes:
        if case["boundary"] == "cpml":
            extra += 5 * _psi_cells(s, case["layers"])
        else:  # one 54-64-64-6 network per outer cell
            outer = s[0] * s[1] * s[2] - (s[0] - 2) * (s[1] - 2) * (s[2] - 2)
            extra += 2 * outer * (54 * 64 + 64 * 64 + 64 * 6)
    return {"bytes": 28 * cells, "flops": (36 * cells + extra) * steps}


def _batch_sizes(case):
    sizes, pad, out = random.Random(5), 2 * case["layers"], []
    for _ in range(case["grids"]):
        if sizes.random() < 0.5:
            s = (sizes.randint(case["lo"], case["hi"]),) * 3
        else:
            s = tuple(sizes.randint(case["lo"], case["hi"]) for _ in range(3))
        s = tuple(n + pad for n in s)
        out.append((s[0], s[1], -(-s[2] // 4) * 4))
    return out


# ------------------------------------------------------- the same in 64 bits


def _f32(v):
    return float(np.float32(v))


def _sigma(n, layers, dx):
    s = np.zeros(n)
    for i in range(layers):
        v = 0.8 * 4.0 / dx * ((layers - i) / layers)**3
        s[i] = v
        s[n - 1 - i] = v
    return s


def _along(v, axis, dims):
    shape = [1] * dims
    shape[axis] = -1
    return torch.as_tensor(v, dtype=torch.float64, device="cuda").reshape(shape)


def _pulse(s, steps, dt):
    """Gaussian-modulated sine, delayed four widths, or a plain sine."""
    if s["width"] is None:
        return np.sin(2.0 * np.pi * s["frequency"] * (np.arange(steps) * dt))
    u = np.arange(steps) * dt - 4.0 * s["width"] * dt
    return np.exp(-(u / (s["width"] * dt))**2) * np.sin(2.0 * np.pi * s["frequency"] * u)


class _Yee:
    """3D Yee step on FP64 tensors, out of place (autograd goes through it)."""

    def __init__(self, size, dx, boundary, layers, eps, kappa_max=1.0, alpha_max=0.0):
        self.size, self.boundary, self.dt = size, boundary, _dt(dx, 3)
        dt = self.dt
        one = [torch.ones(n, dtype=torch.float64, device="cuda") for n in size]
        lo, hi = [v.clone() for v in one], [v.clone() for v in one]
        if boundary != "periodic":
            for k in range(3):
                hi[k][-1] = 0.0  # H is not updated on the last index of its differencing axes
                lo[k][0] = 0.0   # E is not updated on the first
        pairs = ((1, 2), (2, 0), (0, 1))
        a = dt / (MU0 * dx)
        self.am = [a * _along(hi[p], p, 3) * _along(hi[q], q, 3) for p, q in pairs]
        cb = dt / (EPS0 * dx) / (eps if eps is not None else 1.0)
        self.cbm = [cb * _along(lo[p], p, 3) * _along(lo[q], q, 3) for p, q in pairs]
        self.damp = None
        if boundary == "absorbing":
            s = sum(_along(_sigma(n, layers, dx), k, 3) for k, n in enumerate(size)) / 3.0
            self.damp = torch.exp(-s * dt / EPS0)
        self.tab = None
        if boundary == "cpml":
            self.tab = []
            eta0 = math.sqrt(MU0 / EPS0)
            smax = -4.0 * math.log(1e-6) / (2.0 * eta0 * layers * dx)
            for k, n in enumerate(size):
                t = {}
                for name, off in (("e", 0.0), ("h", 0.5)):
                    x = np.arange(n) + off
                    rho = np.clip(np.maximum((layers - x) / layers, (x - (n - 1 - layers)) / layers),
                                  0.0, 1.0)
                    sig = smax * rho**3
                    kap = 1.0 + (kappa_max - 1.0) * rho**3
                    alp = np.where(rho > 0, alpha_max * (1.0 - rho), 0.0)
                    b = np.exp(-(sig / kap + alp) * dt / EPS0)
                    den = sig * kap + kap**2 * alp
                    c = np.where(sig > 0, sig * (b - 1.0) / np.where(den > 0, den, 1.0), 0.0)
                    t[name] = [_along(v, k, 3) for v in (b, c, 1.0 / kap)]
                self.tab.append(t)
        self.stretched = kappa_max != 1.0

    def zeros(self):
        z = lambda: torch.zeros(self.size, dtype=torch.float64, device="cuda")  # noqa: E731
        return [z() for _ in range(6)], [z() for _ in range(12 if self.tab else 0)]

    def _half(self, f, psi, where, shift, sign, base):
        """The curl of (f0, f1, f2) with one-sided differences."""
        curl = []
        for c, (p, q) in enumerate(((1, 2), (2, 0), (0, 1))):
            # component c: d f[q] / d p  -  d f[p] / d q
            d1 = sign * (torch.roll(f[q], shift, p) - f[q])
            d2 = sign * (torch.roll(f[p], shift, q) - f[p])
            if self.tab is None:
                curl.append(d1.sub_(d2) if not d1.requires_grad else d1 - d2)
                continue
            b1, c1, k1 = self.tab[p][where]
            b2, c2, k2 = self.tab[q][where]
            psi[base + 2 * c] = torch.addcmul(b1 * psi[base + 2 * c], c1, d1)
            psi[base + 2 * c + 1] = torch.addcmul(b2 * psi[base + 2 * c + 1], c2, d2)
            if self.stretched:
                d1, d2 = k1 * d1, k2 * d2
            curl.append((d1 - d2) + (psi[base + 2 * c] - psi[base + 2 * c + 1]))
        return curl

    def step(self, f, psi, sources):
        """sources: (component, flat cells, values) of this step."""
        f, psi = list(f), list(psi)
        cu = self._half(f[:3], psi, "h", -1, 1.0, 0)
        for c in range(3):
            f[3 + c] = torch.addcmul(f[3 + c], self.am[c], cu[c], value=-1.0)
        cu = self._half(f[3:], psi, "e", 1, -1.0, 6)
        for c in range(3):
            f[c] = torch.addcmul(f[c], self.cbm[c], cu[c])
            if self.damp is not None:
                f[c] = f[c] * self.damp
        for c, cells, v in sources:
            f[c] = f[c].reshape(-1).index_add(0, cells, v).reshape(self.size)
        return f, psi


def _cells(size, positions):
    return torch.tensor([(x * size[1] + y) * size[2] + z for x, y, z in positions], device="cuda")


def _exact2d(case, seed):
    sources, walls = _spec2d(case, seed)
    nx, ny, dx = case["nx"], case["ny"], 0.01
    dt = _dt(dx, 2)
    a, b = dt / (MU0 * dx), dt / (EPS0 * dx)
    ez, hx, hy = (torch.zeros((nx, ny), dtype=torch.float64, device="cuda") for _ in range(3))
    sig = 0.5 * (_along(_sigma(nx, 10, dx), 0, 2) + _along(_sigma(ny, 10, dx), 1, 2))
    damp = torch.exp(-sig * dt / EPS0)
    keep = torch.ones((nx, ny), dtype=torch.float64, device="cuda")
    for y, g0, g1 in walls:
        keep[:, y] = 0.0
        keep[g0:g1, y] = 1.0
    frames = {k: [] for k in FIELDS2D}
    bnd = case["boundary"]
    for n in range(case["steps"]):
        if bnd == "periodic":
            hx -= a * (torch.roll(ez, -1, 1) - ez)
            hy += a * (torch.roll(ez, -1, 0) - ez)
            ez += b * ((hy - torch.roll(hy, 1, 0)) - (hx - torch.roll(hx, 1, 1)))
        else:
            hx[:, :-1] -= a * (ez[:, 1:] - ez[:, :-1])
            hy[:-1] += a * (ez[1:] - ez[:-1])
            ez[1:, 1:] += b * ((hy[1:, 1:] - hy[:-1, 1:]) - (hx[1:, 1:] - hx[1:, :-1]))
        if bnd == "absorbing":
            ez *= damp
        else:
            near, far = (1, -2) if bnd == "reflecting" else (-2, 1)
            for f in (ez, hx, hy):
                f[0] = f[near]
                f[-1] = f[far]
                f[:, 0] = f[:, near]
                f[:, -1] = f[:, far]
        for freq, y, amp in sources:
            ez[:, y] += _f32(amp) * math.sin(2.0 * math.pi * freq * (n * dt))
        ez *= keep
        if n % case["save_every"] == 0:
            for k, f in zip(FIELDS2D, (ez, hx, hy)):
                frames[k].append(f.clone())
    return {k: torch.stack(v) for k, v in frames.items()}


def _exact3d(case, seed):
    sources, boxes = _spec3d(case, seed)
    size, dx = (case["nx"], case["ny"], case["nz"]), 0.01
    eps = None
    if boxes:
        eps = torch.ones(size, dtype=torch.float64, device="cuda")
        for a, b, e in boxes:
            eps[a[0]:b[0], a[1]:b[1], a[2]:b[2]] = e
    yee = _Yee(size, dx, case["boundary"], case["layers"], eps)
    f, psi = yee.zeros()
    at = [(POL[pol], _cells(size, [pos]), _f32(amp), freq) for freq, pos, amp, pol in sources]
    frames = [[] for _ in range(6)]
    for n in range(case["steps"]):
        src = [(c, i, torch.tensor([amp * math.sin(2.0 * math.pi * freq * (n * yee.dt))],
                                   dtype=torch.float64, device="cuda")) for c, i, amp, freq in at]
        f, psi = yee.step(f, psi, src)
        if n % case["save_every"] == 0:
            for c in range(6):
                frames[c].append(f[c])
    return {k: torch.stack(v) for k, v in zip(FIELDS3D, frames)}


def _run_sources(yee, sources, cells, comps, steps):
    at = [(POL[s["polarization"]], _cells(yee.size, [s["position"]]),
           torch.from_numpy(_f32(s["amplitude"]) * _pulse(s, steps, yee.dt)).cuda()) for s in sources]
    f, psi = yee.zeros()
    traces = torch.zeros((steps, len(comps)), dtype=torch.float64, device="cuda")
    for n in range(steps):
        f, psi = yee.step(f, psi, [(c, i, wave[n:n + 1]) for c, i, wave in at])
        for k, (cell, comp) in enumerate(zip(cells, comps)):
            traces[n, k] = f[comp].view(-1)[cell]
    return traces, f


def _exact_run(case, seed):
    sources, probes, eps = _spec_run(case, seed)
    size = (case["nx"], case["ny"], case["nz"])
    kw = dict(kappa_max=5.0, alpha_max=0.02) if case["stretched"] else {}
    yee = _Yee(size, 1.0, "cpml", case["layers"], None if eps is None else eps.double(), **kw)
    cells = [int(i) for i in _cells(size, [p for p, _ in probes])]
    traces, f = _run_sources(yee, sources, cells, [FIELDS3D.index(c) for _, c in probes],
                            case["steps"])
    return {"traces": traces, **dict(zip(FIELDS3D, f))}


def _exact_batch(case, seed):
    if case["boundary"] == "learned":
        return None  # the band is a 16-bit network: it has no value in 64 bits
    traces, fields = [], [[] for _ in range(6)]
    for size, eps, source in _spec_batch(case, seed):
        yee = _Yee(size, 1.0, "cpml", case["layers"], eps.double())
        cell = int(_cells(size, [tuple(p + 3 for p in source["position"])])[0])
        t, f = _run_sources(yee, [source], [cell], [2], case["steps"])
        traces.append(t.reshape(-1))
        for c in range(6):
            fields[c].append(f[c].reshape(-1))
    return {"traces": torch.cat(traces), **{k: torch.cat(v) for k, v in zip(FIELDS3D, fields)}}


def _exact_adjoint(case, seed):
    """Reverse mode through every step, in segments restarted from saved states."""
    eps, source, probe = _spec_adjoint(case, seed)
    n, steps = case["n"], case["steps"]
    size = (n, n, n)
    eps = eps.detach().double().requires_grad_(True)
    wave = torch.from_numpy(_f32(source["amplitude"]) * _pulse(source, steps, _dt(1.0, 3))).cuda()
    plane = _cells(size, [(i, j, source["z"]) for i in range(n) for j in range(n)])
    cell = int(_cells(size, [probe])[0])
    every = max(1, int(math.sqrt(steps)))

    def advance(yee, f, psi, lo, hi):
        out = []
        for k in range(lo, hi):
            f, psi = yee.step(f, psi, [(0, plane, wave[k].expand(n * n))])
            out.append(torch.stack([f[2].reshape(-1)[cell], f[0].reshape(-1)[cell]]))
        return f, psi, torch.stack(out)

    saved, traces = [], []
    with torch.no_grad():
        yee = _Yee(size, 1.0, case["boundary"], case["layers"], eps)
        f, psi = yee.zeros()
        for lo in range(0, steps, every):
            saved.append((f, psi))
            f, psi, t = advance(yee, f, psi, lo, min(lo + every, steps))
            traces.append(t)
    traces = torch.cat(traces)
    total, after = torch.zeros_like(eps), None
    for s in range(len(saved) - 1, -1, -1):
        lo, hi = s * every, min((s + 1) * every, steps)
        state = [v.detach().requires_grad_(True) for v in saved[s][0] + saved[s][1]]
        yee = _Yee(size, 1.0, case["boundary"], case["layers"], eps)
        f, psi, t = advance(yee, state[:6], state[6:], lo, hi)
        ends, grads = [t], [2.0 * traces[lo:hi]]
        if after is not None:
            pairs = [(e, g) for e, g in zip(f + psi, after) if g is not None]
            ends += [e for e, _ in pairs]
            grads += [g for _, g in pairs]
        got = torch.autograd.grad(ends, [eps] + state, grads, allow_unused=True)
        total += got[0]
        after = got[1:]
    return {"traces": traces, "grad": total}


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid2d":
        return _exact2d(case, seed)
    if kind == "grid3d":
        return _exact3d(case, seed)
    if kind == "run3d":
        return _exact_run(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return _exact_batch(case, seed)
