"""Performance cases: what a user of this package has it compute, through its public entry points.

A case is one call, or one stretch of calls, that a user's program makes again and again:

* ``run``: ``Simulation.run()``, host scene in, ``Result`` out (tables, engine, stepping, read-back);
* ``step``: an engine in hand advances through a long run, one stretch of steps at a time, reads its
  monitors and writes a checkpoint to device memory after each;
* ``grad3d``: ``adjoint.value_and_grad_eps`` of one scene;
* ``batch``: ``batch.value_and_grad_eps`` of a batch of uneven 2D TE design instances;
* ``train`` / ``infer``: a training step of the surrogate network, and its objective and gradient
  for a handful of designs.

``exact`` restates the same quantities in float64 with torch operations only.
"""
import math
import os

import numpy as np
import torch

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200 import surrogate as S
from photonfdtd_b200 import workloads as W
from photonfdtd_b200.adjoint import value_and_grad_eps
from photonfdtd_b200.batch import BatchTE
from photonfdtd_b200.batch import value_and_grad_eps as batch_value_and_grad
from photonfdtd_b200.engine import B200Engine, build_tables

C0 = 299_792_458.0
MU0 = 1.256_637_062_12e-6
EPS0 = 8.854_187_8128e-12
PML = 12
_WEIGHTS = os.path.join(os.path.dirname(pf.__file__), "data", "surrogate_config5.npz")


def listed():
    return [
        # the plain 2D scene of a first script: double precision, a field frame every 20 steps
        dict(name="2d tm frames f64", kind="run", nx=104, ny=104, nz=1, cell=50e-9, steps=1712,
             precision="float64", media="dielectric", boxes=2, mon="frames"),
        # a 2D metal / Lorentz structure with spectra and transmission, odd sizes
        dict(name="2d dispersive spectra", kind="run", nx=331, ny=217, nz=1, cell=20e-9, steps=900,
             precision="float32", media="dispersive", boxes=5, mon="dft+flux"),
        # a small 3D device in double precision with plane frames
        dict(name="3d small frames f64", kind="run", nx=61, ny=53, nz=47, cell=40e-9, steps=500,
             precision="float64", media="dielectric", boxes=3, mon="plane frames"),
        # an ordinary 3D plasmonic run from scene to spectra
        dict(name="3d dispersive blocks", kind="run", nx=128, ny=128, nz=128, cell=10e-9, steps=800,
             precision="float32", media="blocks", boxes=0, mon="dft+flux"),
        # stepping with the diagonal tensor (one coefficient per component), odd sizes, 16 wavelengths
        dict(name="3d tensor steps", kind="step", nx=301, ny=287, nz=263, cell=20e-9, steps=40,
             precision="float32", media="tensor", boxes=8, mon="dft16"),
        # the float64 shadow of a 3D run (error statements are made with it)
        dict(name="3d dielectric steps f64", kind="step", nx=160, ny=152, nz=144, cell=20e-9, steps=40,
             precision="float64", media="dielectric", boxes=8, mon="dft"),
        # the headline workload: 384^3 dispersive blocks, six flux planes and a DFT every step
        dict(name="3d dispersive steps 384", kind="step", nx=384, ny=384, nz=384, cell=10e-9, steps=40,
             precision="float32", media="blocks", boxes=0, mon="dft+flux"),
        # the gradient of a spectral objective with respect to every cell of a 3D scene
        dict(name="3d gradient", kind="grad3d", nx=97, ny=89, nz=101, cell=20e-9, steps=200,
             precision="float32", media="dielectric", boxes=4, mon="dft"),
        # a few inverse-design candidates, many steps
        dict(name="2d batch gradient 8", kind="batch", inst=8, steps=1800, lo=0, precision="float32"),
        # a whole population of candidates
        dict(name="2d batch gradient 256", kind="batch", inst=256, steps=1200, lo=0, precision="float32"),
        # surrogate training at its usual batch size
        dict(name="surrogate training step", kind="train", batch=128),
        # surrogate objective and gradient of the designs of one optimiser step
        dict(name="surrogate gradient", kind="infer", batch=32, n=27),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run2d", "run2d", "run3d", "step", "step", "grad3d", "batch", "batch", "train", "infer"])
    if kind == "run2d":
        media = rng.choice(["dielectric", "dispersive"])
        return dict(kind="run", nx=_log(rng, 60, 420), ny=_log(rng, 60, 420), nz=1,
                    cell=rng.choice([20e-9, 50e-9]), steps=_log(rng, 200, 1600),
                    precision=rng.choice(["float32", "float64"]),
                    media=media, boxes=rng.randint(1, 6), mon=rng.choice(["frames", "dft+flux"]))
    if kind == "run3d":
        return dict(kind="run", nx=_log(rng, 40, 128), ny=_log(rng, 40, 128), nz=_log(rng, 40, 128),
                    cell=rng.choice([10e-9, 20e-9]), steps=_log(rng, 100, 700),
                    precision=rng.choice(["float32", "float32", "float64"]),
                    media=rng.choice(["dielectric", "dispersive", "blocks"]), boxes=rng.randint(1, 6),
                    mon=rng.choice(["plane frames", "dft+flux"]))
    if kind == "step":
        media = rng.choice(["dielectric", "blocks", "tensor"])
        f64 = rng.random() < 0.25
        hi = 200 if f64 else 340
        return dict(kind="step", nx=_log(rng, 96, hi), ny=_log(rng, 96, hi), nz=_log(rng, 96, hi),
                    cell=10e-9 if media == "blocks" else 20e-9, steps=rng.randint(12, 40),
                    precision="float64" if f64 else "float32", media=media, boxes=rng.randint(1, 8),
                    mon=rng.choice(["dft", "dft16", "dft+flux"]))
    if kind == "grad3d":
        return dict(kind="grad3d", nx=_log(rng, 40, 110), ny=_log(rng, 40, 110), nz=_log(rng, 40, 110),
                    cell=20e-9, steps=_log(rng, 60, 200), precision="float32", media="dielectric",
                    boxes=rng.randint(1, 5), mon="dft")
    if kind == "batch":
        n = _log(rng, 4, 96)
        return dict(kind="batch", inst=n, steps=_log(rng, 1100, 1800), lo=rng.randint(0, 256 - n),
                    precision="float32")
    if kind == "train":
        return dict(kind="train", batch=32 * _log(rng, 1, 4))
    b = 32 * rng.randint(1, 4)
    return dict(kind="infer", batch=b, n=rng.randint(max(1, b - 31), b))


# --------------------------------------------------------------------------- #
# Scenes
# --------------------------------------------------------------------------- #
def _dims(c):
    return [c["nx"], c["ny"], c["nz"]]


def _dt(c):
    nd = sum(n > 1 for n in _dims(c))
    return 0.99 / (C0 * math.sqrt(nd / c["cell"] ** 2))


def _scene(c, seed):
    """Random numbers of a scene, as plain values both `prepare` and `exact` read."""
    r = np.random.default_rng(seed)
    d, n = c["cell"], _dims(c)
    boxes = []
    for q in range(c["boxes"]):
        # box faces on half-integer cell positions, inside the absorbing layers
        lo, hi = [], []
        for m in n:
            if m == 1:
                lo.append(0)
                hi.append(1)
                continue
            w = int(r.integers(4, max(5, (m - 2 * PML) // 2)))
            a = int(r.integers(PML, m - PML - w + 1))
            lo.append(a)
            hi.append(a + w)
        boxes.append((lo, hi, float(r.uniform(1.5, 12.1))))
    lam = 25.0 * d * float(r.uniform(0.9, 1.1))
    src = [m // 2 + (int(r.integers(-4, 5)) if m > 1 else 0) for m in n]
    freqs = C0 / (lam * np.linspace(0.92, 1.08, 16 if c["mon"] == "dft16" else 8))
    ids = r.integers(0, 3, size=tuple(-(-m // 8) for m in n)) if c["media"] == "blocks" else None
    fwhm = 60.0 * _dt(c)  # the pulse is over well inside the run
    tensor = r.uniform(0.9, 1.1, size=3)
    comp = ("Ez" if c["media"] == "dielectric" else "Ey") if c["nz"] == 1 else "Ex"
    return dict(boxes=boxes, f0=C0 / lam, fwhm=fwhm, src=src, freqs=freqs, ids=ids, comp=comp, tensor=tensor)


def _media(c):
    """Drude metal and two-pole Lorentz medium: (eps_inf, [(strength, omega0, gamma)]), resolved alike
    at every cell size (the plasma frequency times dt is 0.26, as for gold at 10 nm)."""
    u = 0.26 / 1.37e16 / _dt(c)
    return [(1.0, [((1.37e16 * u) ** 2, 0.0, 1.0e14 * u)]),
            (1.0, [((3e15 * u) ** 2, 3e15 * u, 1e13 * u), (0.5 * (6e15 * u) ** 2, 6e15 * u, 1e13 * u)])]


def _cells(c, s):
    """(eps, medium) grids: relative permittivity and dispersive medium (-1: none) per cell."""
    n = _dims(c)
    eps, med = np.ones(n), np.full(n, -1, np.int8)
    if c["media"] == "blocks":
        b = np.repeat(np.repeat(np.repeat(s["ids"], 8, 0), 8, 1), 8, 2)[:n[0], :n[1], :n[2]]
        eps[b == 2] = 2.1
        med[b == 0] = 0
        med[b == 1] = 1
        return eps, med
    for q, (lo, hi, e) in enumerate(s["boxes"]):
        sl = tuple(slice(a, b) for a, b in zip(lo, hi))
        m = q % 3 if c["media"] == "dispersive" else 2
        eps[sl] = e if m == 2 else _media(c)[m][0]
        med[sl] = -1 if m == 2 else m
    return eps, med


def _planes(c):
    """Flux planes (axis, index) and the DFT plane (axis, index)."""
    n = _dims(c)
    if c["nz"] == 1:
        return [(0, n[0] // 4), (0, 3 * n[0] // 4), (1, n[1] // 3)], (0, n[0] - 20)
    return [(a, i) for a in range(3) for i in (n[a] // 4, 3 * n[a] // 4)], (2, n[2] // 2)


def _dft_comps(c):
    if c["nz"] == 1:
        return ("Ez", "Hy") if c["media"] == "dielectric" else ("Ey", "Hz")
    return ("Ex", "Ey", "Hx", "Hy") if c["mon"] == "dft16" else ("Ex", "Ey")


def _every(c):
    return 20 if c["nz"] == 1 else 25


def _run_steps(c):
    """Steps of the whole run that a case's scene belongs to: a `step` case advances through a long one."""
    if c["kind"] != "step":
        return c["steps"]
    cells = float(np.prod(_dims(c)))
    return c["steps"] * (1200 if cells < 2e6 else 600 if cells < 8e6 else 250)


def _simulation(c, s):
    d, n = c["cell"], _dims(c)
    size = tuple(m * d if m > 1 else 0.0 for m in n)
    grid = pf.Grid(size=size, cell_size=tuple(d if m > 1 else 0.0 for m in n), pml_layers=tuple(PML if m > 1 else 0 for m in n))
    structures = []
    media = [pf.DispersiveMedium(eps_inf=e, poles=tuple(pf.Pole(strength=a, omega0=b, gamma=g) for a, b, g in p))
             for e, p in _media(c)]
    if c["media"] == "blocks":
        structures = [W.BlockMedium(m, s["ids"], q, 8)
                      for q, m in enumerate(media + [pf.Medium(permittivity=2.1)])]
    else:
        for q, (lo, hi, e) in enumerate(s["boxes"]):
            m = media[q % 3] if c["media"] == "dispersive" and q % 3 < 2 else pf.Medium(permittivity=e)
            ctr = tuple(((a + b - 1) / 2 - (k - 1) / 2) * d if k > 1 else 0.0 for a, b, k in zip(lo, hi, n))
            structures.append(pf.Box(center=ctr, size=tuple((b - a) * d for a, b in zip(lo, hi)), medium=m))
    at = tuple(float(co[i]) for co, i in zip(grid.coords, s["src"]))
    src = pf.PointDipole(position=at, component=s["comp"], waveform=pf.GaussianPulse(freq0=s["f0"], fwhm=s["fwhm"]))
    mons = []
    if c["mon"] == "frames":
        mons.append(pf.FieldMonitor(name="m", components=(s["comp"],), interval=_every(c)))
    elif c["mon"] == "plane frames":
        mons.append(pf.FieldMonitor(name="m", components=("Ex", "Hz"), interval=_every(c),
                                    plane_z=float(grid.coords[2][n[2] // 2])))
    else:
        flux, (ax, idx) = _planes(c)
        mons.append(pf.DFTMonitor(name="d", components=_dft_comps(c), freqs=s["freqs"], plane_axis="xyz"[ax],
                                  plane_position=float(grid.coords[ax][idx])))
        if "flux" in c["mon"]:
            for q, (a, i) in enumerate(flux):
                mons.append(pf.FluxMonitor(name="f%d" % q, plane_axis="xyz"[a], plane_position=float(grid.coords[a][i])))
    return pf.Simulation(grid, structures=structures, sources=[src], monitors=mons,
                         run_time=(_run_steps(c) - 0.5) * _dt(c), precision=c["precision"])


def _tensor_ce(c, s):
    """Per-component coefficients dt / (eps_c eps0) of a mildly anisotropic scene."""
    eps, _ = _cells(c, s)
    return [_dt(c) / (np.where(eps > 1.0, eps * t, 1.0) * EPS0) for t in s["tensor"]]


def _start_fields(c, seed):
    """Smooth random fields in the field type: a few standing waves of about 20 cells' wavelength."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n, dev = _dims(c), "cuda"
    ty = torch.float64 if c["precision"] == "float64" else torch.float32
    out = torch.zeros([6] + n, dtype=ty, device=dev)
    for f in range(6):
        for _ in range(3):
            w = 1.0
            for a in range(3):
                k, p = torch.rand(2, generator=g, device=dev, dtype=torch.float64)
                x = torch.arange(n[a], device=dev, dtype=torch.float64)
                v = torch.sin(x * (0.2 + 0.15 * k) + 6.28 * p)
                # fields that fade out before the absorbing layers
                edge = torch.clamp((torch.minimum(x, n[a] - 1 - x) - PML) / 10.0, 0.0, 1.0)
                shape = [1, 1, 1]
                shape[a] = n[a]
                w = w * (v * edge).reshape(shape).to(ty)
            out[f] += w * (1.0 if f < 3 else 1.0 / 377.0)
    return out


# --------------------------------------------------------------------------- #
# prepare / run
# --------------------------------------------------------------------------- #
def _batch_rho(i, seed, n=64):
    """A smooth random density in (0, 1)."""
    r = np.random.default_rng([seed, i])
    k = np.fft.fftfreq(n)
    h = np.exp(-2.0 * (math.pi * 3.0) ** 2 * (k[:, None] ** 2 + k[None, :] ** 2))
    g = np.fft.ifft2(np.fft.fft2(r.standard_normal((n, n))) * h).real
    return 1.0 / (1.0 + np.exp(-g / g.std()))


def _batch_sizes(c):
    return W.config4_sizes(256)[c["lo"]:c["lo"] + c["inst"]]


def _designs(n, seed):
    return np.stack([_batch_rho(i, seed) for i in range(n)]).astype(np.float32)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "run" or kind == "grad3d":
        return dict(kind=kind, sim=_simulation(c, _scene(c, seed)))
    if kind == "step":
        s = _scene(c, seed)
        sim = _simulation(c, s)
        t = build_tables(sim, ce3=_tensor_ce(c, s) if c["media"] == "tensor" else None)
        fields = _start_fields(c, seed)
        n, layer = _dims(c), [[int(np.count_nonzero(q[k])) for q in t["cpml"]] for k in (1, 3)]
        psi = sum(2 * fields[0].numel() // n[a] * m[a] for m in layer for a in range(3))
        state = dict(kind=kind, tables=t, fields=fields, steps=c["steps"], shape=list(fields.shape), psi=psi)
        _new_run(state)
        return state
    if kind == "batch":
        sims, windows = [], []
        rho0 = np.zeros((64, 64))
        for nx, ny in _batch_sizes(c):
            sims.append(W.config4_instance(pf, nx, ny, rho=rho0, n_steps=c["steps"], precision=c["precision"]))
            windows.append(W.design_window_box(nx, ny, 64))
        b = BatchTE(sims, windows)
        eps = W.EPS_CLAD + _designs(c["inst"], seed).astype(np.float64) * (W.EPS_CORE - W.EPS_CLAD)
        return dict(kind=kind, batch=b, eps=eps.reshape(-1))
    net = S.SurrogateNet.load(_WEIGHTS, batch=c["batch"])
    if kind == "train":
        g = torch.Generator().manual_seed(int(seed))
        x = torch.from_numpy(2.0 * _designs(c["batch"], seed) - 1.0).cuda()
        t = torch.randn(c["batch"], S.N_FREQ, 2, generator=g).cuda()
        return dict(kind=kind, net=net, x=x, t=t)
    return dict(kind=kind, net=net, rho=_designs(c["n"], seed))


def _new_run(state):
    """An engine at step 0 of the run, with the start fields and zero CPML and polarisation state."""
    eng, f = B200Engine(state["tables"]), state["fields"].reshape(-1)
    out = torch.zeros(eng.state_bytes(), dtype=torch.uint8, device="cuda")
    out.view(f.dtype)[:f.numel()] = f
    torch.cuda.synchronize()
    N.check(N.lib().pf_set_state(eng.h, 0, out.data_ptr(), out.numel(), 1), eng.h)
    state.update(eng=eng, out=out, at=0)


def _grad_loss(out):
    return sum((v.abs() ** 2).sum() for v in out["dft"]["d"].values())


def run(state):
    kind = state["kind"]
    if kind == "run":
        r = state["sim"].run()
        return dict(fields=r.fields, dft=r.dft, flux=r.flux)
    if kind == "step":
        if state["at"] + state["steps"] > state["tables"]["n_steps"]:
            _new_run(state)  # the run is over: the next one
        eng, t = state["eng"], state["tables"]
        eng.advance(state["at"], state["steps"])
        state["at"] += state["steps"]
        eng.get_state_to(state["out"].data_ptr(), state["out"].numel())
        f = state["out"].view(state["fields"].dtype)
        m = int(np.prod(state["shape"]))
        dft = {q: eng.read_dft(0, q, t["dft"][0]["omega"].size, t["dft"][0]["counts"])
               for q in t["dft"][0]["m"].components}
        return dict(fields=f[:m].view(state["shape"]), psi=f[m:m + state["psi"]], dft=dft,
                    flux=[eng.read_flux(k) for k in range(len(t["flux"]))])
    if kind == "grad3d":
        v, g = value_and_grad_eps(state["sim"], _grad_loss)
        return dict(value=v, grad=g)
    if kind == "batch":
        v, g = batch_value_and_grad(state["batch"], state["eps"])
        return dict(value=v, grad=g)
    net = state["net"]
    if kind == "train":
        y = net.forward(state["x"])
        net.loss_grad(state["t"])
        net.backward()
        net.adam_step(1e-3)
        live = [k for k, L in enumerate(net.layers) if L.kind != "up"]
        return dict(y=y, gw=[net.gw[k] for k in live], gb=[net.gb[k] for k in live],
                    w=[net.w32[k] for k in live], b=[net.b32[k] for k in live])
    v, g = net.value_and_grad(state["rho"], S.band_objective)
    return dict(value=v, grad=g)


# --------------------------------------------------------------------------- #
# work
# --------------------------------------------------------------------------- #
def work(case):
    """Bytes: every field read and written once per step, the coefficients and the polarisation state
    likewise, for the components that the grid's dimension couples (three in 2D)."""
    c = case
    if c["kind"] in ("train", "infer"):
        macs, params = 0, 0
        for L in S.plan():
            if L.kind != "up":
                macs += L.Ho * L.Wo * L.cout * L.K
                params += L.cout * (L.K + 1)
        passes = 3 if c["kind"] == "train" else 2
        return dict(bytes=params * (28 if c["kind"] == "train" else 4) + c["batch"] * 64 * 64 * 8,
                    flops=2.0 * passes * macs * c["batch"])
    if c["kind"] == "batch":
        cells = sum(a * b for a, b in _batch_sizes(c))
        # forward and reverse: three fields read and written, one coefficient; the window's curls kept and read
        return dict(bytes=c["steps"] * (2.0 * cells * 28 + c["inst"] * 64 * 64 * 16), flops=c["steps"] * cells * 40.0)
    b = 8 if c["precision"] == "float64" else 4
    cells = int(np.prod(_dims(c)))
    two = c["nz"] == 1
    per = (3 if two else 6) * 2 * b
    per += 3 * b if c["media"] == "tensor" else 4
    if c["media"] == "blocks":
        per += 1.0 * 9 * b  # one pole per cell on average: three components, P^n and P^(n-1) read, one written
    fl = (15 if two else 36)
    if c["kind"] == "grad3d":  # forward, replay with a record, reverse with the record and a gradient
        return dict(bytes=c["steps"] * cells * (3.0 * per + 2 * 12 + 16), flops=c["steps"] * cells * 4.0 * fl)
    return dict(bytes=float(c["steps"]) * cells * per, flops=float(c["steps"]) * cells * fl)


# --------------------------------------------------------------------------- #
# exact: the same quantities in float64 with torch operations
# --------------------------------------------------------------------------- #
def _cpml(n, d, dt):
    """(b_e, c_e, b_h, c_h) of one axis: cubic conductivity grading, 1e-7 target reflection."""
    if n == 1:
        return [np.zeros(1)] * 4
    eta = math.sqrt(MU0 / EPS0)
    smax = 0.8 * 4.0 * -math.log(1e-7) / (2.0 * eta * PML * d)
    tabs = []
    for off in (0.0, 0.5):
        x = np.arange(n) + off
        u = np.zeros(n)
        u[:PML] = np.clip((PML - 1 - x[:PML]) / (PML - 1), 0.0, 1.0)
        u[-PML:] = np.clip((x[-PML:] - (n - PML)) / (PML - 1), 0.0, 1.0)
        on = np.zeros(n, bool)
        on[:PML] = on[-PML:] = True
        sg, al = smax * u ** 3, 0.24 * (1.0 - u)
        b = np.exp(-(sg + al) * dt / EPS0)
        tabs += [np.where(on, b, 0.0), np.where(on, sg / (sg + al) * (b - 1.0), 0.0)]
    return tabs


class _Yee:
    """A float64 Yee grid with CPML and dispersion in plain torch operations, functional per step."""

    def __init__(self, n, d, dt, K, E=None, H=None):
        self.n, self.d, self.dt, self.K = n, d, dt, K
        z = lambda: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
        self.E = E or [z() for _ in range(3)]
        self.H = H or [z() for _ in range(3)]
        self.tab = []
        for a in range(3):
            sh = [1, 1, 1]
            sh[a] = n[a]
            self.tab.append([torch.from_numpy(np.ascontiguousarray(v)).cuda().reshape(sh) for v in _cpml(n[a], d, dt)])
        self.psi = {}
        self.ade = []

    def disperse(self, med, media):
        for m, (einf, poles) in enumerate(media):
            idx = torch.from_numpy(np.flatnonzero(med.reshape(-1) == m)).cuda()
            if idx.numel():
                p = [[torch.zeros(3, idx.numel(), dtype=torch.float64, device="cuda") for _ in range(2)] for _ in poles]
                self.ade.append((idx, einf, poles, p))

    def _curl(self, F, G, K, hi, key):
        """F + K (curl G) with the CPML terms; hi: forward differences (H), else backward (E)."""
        n, out = self.n, []
        for c in range(3):
            a, b = (c + 1) % 3, (c + 2) % 3
            terms = []
            for ax, fld, sign, other in ((a, b, 1.0, b), (b, a, -1.0, a)):
                if n[ax] == 1:
                    continue
                dd = torch.diff(G[fld], dim=ax) / self.d
                if n[other] > 1:
                    dd = dd.narrow(other, 0 if hi else 1, n[other] - 1)
                bb, cc = (self.tab[ax][2 if hi else 0], self.tab[ax][3 if hi else 1])
                bb, cc = (v.narrow(ax, 0 if hi else 1, n[ax] - 1) for v in (bb, cc))
                old = self.psi.get((key, c, ax))
                psi = cc * dd if old is None else bb * old + cc * dd
                self.psi[(key, c, ax)] = psi
                terms.append(sign * (dd + psi))
            if not terms:
                out.append(F[c])
                continue
            t = terms[0] if len(terms) == 1 else terms[0] + terms[1]
            k = K[c]
            pad = []
            for ax in (2, 1, 0):
                r = ax in (a, b) and n[ax] > 1
                pad += [0, 0] if not r else ([0, 1] if hi else [1, 0])
                if torch.is_tensor(k) and r:
                    k = k.narrow(ax, 0 if hi else 1, n[ax] - 1)
            out.append(F[c] + torch.nn.functional.pad(k * t, pad))
        return out

    def step(self, src, val):
        """One step with a soft source val on E component src[0] at cell src[1]."""
        ch = -self.dt / MU0
        self.H = self._curl(self.H, self.E, [ch, ch, ch], True, "h")
        old = self.E
        self.E = self._curl(self.E, self.H, self.K, False, "e")
        for idx, einf, poles, p in self.ade:
            e0 = torch.stack([f.reshape(-1)[idx] for f in old])
            tot = torch.zeros_like(e0)
            for q, (s, w0, g) in enumerate(poles):
                den = 1.0 + g * self.dt
                new = ((2.0 - (w0 * self.dt) ** 2) / den * p[q][0] + (g * self.dt - 1.0) / den * p[q][1]
                       + EPS0 * s * self.dt ** 2 / den * e0)
                tot += new - p[q][0]
                p[q][1], p[q][0] = p[q][0], new
            for k in range(3):
                self.E[k] = self.E[k].contiguous()
                self.E[k].view(-1)[idx] -= tot[k] / (EPS0 * einf)
        for comp, cell, amp in src:
            self.E[comp] = self.E[comp].index_put(cell, torch.as_tensor(val * amp, dtype=torch.float64, device="cuda"), accumulate=True)


def _pulse(f0, fwhm, t):
    sg = fwhm / (2.0 * math.sqrt(2.0 * math.log(2.0)))
    return math.exp(-((t - 4.0 * sg) / sg) ** 2) * math.sin(2.0 * math.pi * f0 * (t - 4.0 * sg))


def _cell(i):
    return tuple(torch.tensor([v], device="cuda") for v in i)


def _march(c, s, y, src):
    """All steps of the case's scene; (frames, dft, flux) of its monitors."""
    n, dt = _dims(c), _dt(c)
    comps = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
    flux, (ax, idx) = _planes(c)
    with_dft = "dft" in c["mon"]
    om = torch.from_numpy(2.0 * np.pi * np.asarray(s["freqs"])).cuda()
    acc, fl, frames = {}, [0.0] * len(flux), {}
    area = [c["cell"] if m > 1 else 1.0 for m in n]
    for k in range(c["steps"]):
        y.step(src, _pulse(s["f0"], s["fwhm"], (k + 1) * dt))
        F = dict(zip(comps, y.E + y.H))
        if with_dft:
            for q in _dft_comps(c):
                ph = torch.exp(1j * om * ((k + (1.0 if q[0] == "E" else 0.5)) * dt)).reshape(-1, 1, 1, 1)
                v = ph * F[q].narrow(ax, idx, 1) * dt
                acc[q] = v if q not in acc else acc[q] + v
        if "flux" in c["mon"]:
            for q, (a, i) in enumerate(flux):
                t1, t2 = (a + 1) % 3, (a + 2) % 3
                e1, e2, h1, h2 = (v.narrow(a, i, 1) for v in (y.E[t1], y.E[t2], y.H[t1], y.H[t2]))
                fl[q] = fl[q] + (e1 * h2 - e2 * h1).sum() * (area[t1] * area[t2] * dt)
        if "frames" in c["mon"] and k % _every(c) == 0:
            for q in ((s["comp"],) if c["mon"] == "frames" else ("Ex", "Hz")):
                v = F[q] if c["mon"] == "frames" else F[q].narrow(2, n[2] // 2, 1)
                frames.setdefault(q, []).append(v)
    fl = [float(v) for v in fl] if "flux" in c["mon"] else []
    return {q: torch.stack(v) for q, v in frames.items()}, acc, fl


def _yee(c, s, eps=None):
    e, med = _cells(c, s)
    e = torch.from_numpy(e).cuda() if eps is None else eps
    K = _dt(c) / (e * EPS0)
    y = _Yee(_dims(c), c["cell"], _dt(c), [K, K, K])
    y.disperse(med, _media(c))
    return y


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch" and c["inst"] * c["steps"] > 15000:
        return None  # minutes of small operations
    if kind in ("run", "step"):
        s = _scene(c, seed)
        y = _yee(c, s)
        comp = ("Ex", "Ey", "Ez").index(s["comp"])
        if kind == "step":
            f = _start_fields(c, seed).double()
            y.E, y.H = [f[0], f[1], f[2]], [f[3], f[4], f[5]]
            if c["media"] == "tensor":
                y.K = [torch.from_numpy(k).cuda() for k in _tensor_ce(c, s)]
        with torch.no_grad():
            frames, acc, fl = _march(c, s, y, [(comp, _cell(s["src"]), 1.0)])
        if kind == "step":
            return dict(fields=torch.stack(y.E + y.H), psi=None, dft={q: v for q, v in acc.items()}, flux=fl)
        return dict(fields={"m": frames} if frames else {}, dft={"d": acc} if acc else {},
                    flux={"f%d" % q: v for q, v in enumerate(fl)})
    if kind == "grad3d":
        s = _scene(c, seed)
        eps = torch.from_numpy(_cells(c, s)[0]).cuda().requires_grad_(True)
        y = _yee(c, s, eps)
        _, acc, _ = _march(c, s, y, [(("Ex", "Ey", "Ez").index(s["comp"]), _cell(s["src"]), 1.0)])
        v = sum((a.abs() ** 2).sum() for a in acc.values())
        v.backward()
        return dict(value=float(v), grad=eps.grad)
    if kind == "batch":
        vals, grads = [], []
        d, dt = 20e-9, 0.99 / (C0 * math.sqrt(2 / 20e-9 ** 2))
        om = torch.from_numpy(2.0 * np.pi * C0 / np.linspace(1.5e-6, 1.6e-6, 8)).cuda()
        rho = _designs(c["inst"], seed).astype(np.float64)
        for i, (nx, ny) in enumerate(_batch_sizes(c)):
            win = torch.from_numpy(W.EPS_CLAD + rho[i] * (W.EPS_CORE - W.EPS_CLAD)).cuda().requires_grad_(True)
            i0, j0 = nx // 2 - 32, ny // 2 - 32
            eps = torch.full((nx, ny), W.EPS_CLAD, dtype=torch.float64, device="cuda")
            eps = torch.nn.functional.pad(win - W.EPS_CLAD, (j0, ny - j0 - 64, i0, nx - i0 - 64)) + eps
            v = _te(nx, ny, d, dt, dt / (eps * EPS0), c["steps"], om)
            v.backward()
            vals.append(float(v))
            grads.append(win.grad.reshape(-1))
        return dict(value=np.array(vals), grad=torch.cat(grads))
    return _exact_net(c, seed)


def _te(nx, ny, d, dt, K, steps, om):
    """sum |DFT of Ey|^2 on the output line of one 2D TE instance driven by its Ey line source."""
    dev = "cuda"
    tx = [torch.from_numpy(np.ascontiguousarray(v)).cuda().reshape(-1, 1) for v in _cpml(nx, d, dt)]
    ty = [torch.from_numpy(np.ascontiguousarray(v)).cuda().reshape(1, -1) for v in _cpml(ny, d, dt)]
    ex = torch.zeros(nx, ny, dtype=torch.float64, device=dev)
    ey, hz = torch.zeros_like(ex), torch.zeros_like(ex)
    pa = torch.zeros(nx - 1, ny - 1, dtype=torch.float64, device=dev)
    pb = torch.zeros_like(pa)
    px, py = torch.zeros(nx, ny - 1, dtype=torch.float64, device=dev), torch.zeros(nx - 1, ny, dtype=torch.float64, device=dev)
    line = torch.zeros(nx, ny, dtype=torch.float64, device=dev)
    line[20, PML:ny - PML] = 1.0
    ch, pad, acc = dt / MU0, torch.nn.functional.pad, 0.0
    ax_h, ay_h = tx[2][:-1], ty[2][:, :-1]
    cx_h, cy_h = tx[3][:-1], ty[3][:, :-1]
    for k in range(steps):
        da = (ey[1:, :-1] - ey[:-1, :-1]) / d
        db = (ex[:-1, 1:] - ex[:-1, :-1]) / d
        pa, pb = ax_h * pa + cx_h * da, ay_h * pb + cy_h * db
        hz = hz - ch * pad(da - db + pa - pb, (0, 1, 0, 1))
        dy = (hz[:, 1:] - hz[:, :-1]) / d
        dx = (hz[1:] - hz[:-1]) / d
        px, py = ty[0][:, 1:] * px + ty[1][:, 1:] * dy, tx[0][1:] * py + tx[1][1:] * dx
        ex = ex + K * pad(dy + px, (1, 0))
        ey = ey - K * pad(dx + py, (0, 0, 1, 0)) + line * _pulse(C0 / 1.55e-6, 15e-15, (k + 1) * dt)
        acc = acc + torch.exp(1j * om * ((k + 1) * dt)).reshape(-1, 1) * ey[nx - 21] * dt
    return (acc.abs() ** 2).sum()


def _exact_net(c, seed):
    layers = S.plan()
    params = S.SurrogateNet.load_params(_WEIGHTS)
    w = [None if p[0] is None else torch.from_numpy(p[0].astype(np.float32)).double().cuda().requires_grad_(True) for p in params]
    b = [None if p[1] is None else torch.from_numpy(p[1].astype(np.float32)).double().cuda().requires_grad_(True) for p in params]
    rho = torch.from_numpy(_designs(c["batch"] if c["kind"] == "train" else c["n"], seed)).double().cuda().requires_grad_(True)
    a = (2.0 * rho - 1.0)[:, None]  # (B, C, H, W)
    n = a.shape[0]
    for L, wi, bi in zip(layers, w, b):
        if L.kind == "up":
            a = a.repeat_interleave(2, dim=3)
            continue
        if L.kind == "conv":
            k = wi.reshape(L.cout, L.kh, L.kw, L.cin).permute(0, 3, 1, 2)
            a = torch.nn.functional.conv2d(a, k, bi, stride=L.stride, padding=(L.ph, L.pw))
        else:
            a = a.permute(0, 2, 3, 1).reshape(n, -1) @ wi.T + bi
            a = a.reshape(n, 1, -1, 64).permute(0, 3, 1, 2)
        a = torch.relu(a) if L.relu else a
    y = a[:, :, 0, :].permute(0, 2, 1)
    if c["kind"] == "infer":
        z = np.load(_WEIGHTS)
        y = y * torch.from_numpy(z["t_std"]).cuda() + torch.from_numpy(z["t_mean"]).cuda()
        T = torch.complex(y[..., 0], y[..., 1])
        v = S.band_objective(T)
        v.sum().backward()
        return dict(value=v.detach(), grad=rho.grad)
    t = torch.randn(n, S.N_FREQ, 2, generator=torch.Generator().manual_seed(int(seed))).double().cuda()
    ((y - t) ** 2).mean().backward()
    out = dict(y=y.detach(), gw=[], gb=[], w=[], b=[])
    for L, wi, bi in zip(layers, w, b):
        if L.kind == "up":
            continue

        def grow(v, shape):
            z = torch.zeros(shape, dtype=torch.float64, device="cuda")
            z[tuple(slice(0, m) for m in v.shape)] = v
            return z
        shapes = ((L.coutp, L.Kp), (L.coutp,))
        for p, sh, g_, v_ in ((wi, shapes[0], "gw", "w"), (bi, shapes[1], "gb", "b")):
            g = p.grad
            new = p.detach() - 1e-3 * g / (g.abs() + 1e-8)
            out[g_].append(grow(g, sh))
            out[v_].append(grow(new, sh))
    return out
