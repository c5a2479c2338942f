"""The workloads by which this framework's speed is judged, over the range of sizes and options it is used for.

A pass of every case is one whole call sequence of a user's program through the public entry points
(SPEContext, Ensemble, solver.SPE3D_waveDM and the operators, autograd.evolve_loss), starting from that pass's
input state.  exact() restates each of them in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

import wavedm_gb300 as wdm
from wavedm_gb300 import autograd, solver

SIZES = (8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)
DEV = "cuda"

# what a step case may set; the values a run has by default
STEP = dict(kind="step", batch=1, mode="strang", phase="precise", grid="periodic", graph=False, tide=False,
            centre="box_centre", baryons=0, kerr=0.0, absorb=0.0, potential=False)


def _step(name, n, steps, box, **options):
    return dict(STEP, name=name, nx=n[0], ny=n[1], nz=n[2], steps=steps, box=box, **options)


def listed():
    return [
        # the smallest calls: a batch of test-size halos advanced by replayed graphs, all latency
        _step("graph_32_batch4", (32, 32, 32), 10, 10.0, batch=4, graph=True),
        # a small single halo (soliton formation runs), stepped between snapshots
        _step("strang_64", (64, 64, 64), 20, 20.0),
        # an ordinary production grid
        _step("strang_256", (256, 256, 256), 10, 30.0),
        # the largest: a satellite halo in its host's time-dependent tide, with a stellar component of 1e5 particles
        _step("strang_384_tide_stars", (384, 384, 384), 10, 40.0, tide=True, baryons=100_000),
        # an oblong box with every optional term, in the literal K(dt/2) D(dt) order of the reference's loop with FP32
        # phases, on its endpoint-inclusive grid
        _step("loop_192x96x48_options", (192, 96, 48), 20, 24.0, mode="reference_loop", phase="plain",
              grid="reference", tide=True, centre="reference", kerr=0.3, absorb=2.0, potential=True),
        # a survey of 128 halos of three grid sizes in one group, each with its own constant tide
        dict(name="ensemble_128_halos", kind="ensemble", groups="64:96,96:24,128:8", steps=5, box=20.0),
        # fitting an initial state and a tidal amplitude to a target density: loss and gradients
        dict(name="adjoint_128", kind="adjoint", nx=128, ny=128, nz=128, steps=40, every=10, box=20.0),
        # what a run does at a snapshot: diagnostics (radii, virial sums, limits), density and potential
        dict(name="snapshot_256", kind="snapshot", nx=256, ny=256, nz=256, box=30.0),
        # the Poisson solve alone, of a density that another code computed on the device (oblong box)
        dict(name="poisson_384x256x192", kind="poisson", nx=384, ny=256, nz=192, box=30.0),
        # the transform alone, of the largest supported grid
        dict(name="fft_512", kind="fft", nx=512, ny=512, nz=512, inverse=False),
        # the whole solver entry, from an array of initial values on the host to the final state on the host
        dict(name="solver_48", kind="solver", nx=48, ny=48, nz=48, steps=40, every=10, box=16.0),
        # a host program that keeps the state itself: upload, one step, download
        dict(name="host_step_256x192x128", kind="host", nx=256, ny=192, nz=128, box=24.0),
    ]


def _draw_axes(rng, low, high, most):
    """Axis lengths with the cell count spread over the logarithm of [low, high]: cubes as well as oblong boxes."""
    while True:
        edge = math.exp(rng.uniform(math.log(low), math.log(high)))
        if rng.random() < 0.4:
            n = (min(SIZES, key=lambda s: abs(math.log(s / edge))),) * 3
        else:
            n = tuple(min(SIZES, key=lambda s: abs(math.log(s / edge / math.exp(rng.uniform(-0.7, 0.7))))) for _ in "xyz")
        if n[0] * n[1] * n[2] <= most:
            return dict(zip(("nx", "ny", "nz"), n))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["graph"] * 2 + ["ensemble", "adjoint", "snapshot", "poisson", "poisson", "fft",
                                                       "fft", "solver", "host", "operators"])
    box = round(rng.uniform(12.0, 40.0), 2)
    if kind in ("step", "graph"):
        graph = kind == "graph"
        n = _draw_axes(rng, 10, 140 if graph else 400, 384 ** 3)
        cells = n["nx"] * n["ny"] * n["nz"]
        c = dict(STEP, box=box, graph=graph, **n)
        c["steps"] = rng.randint(1, max(1, min(30, 8 * 384 ** 3 // cells)))
        c["batch"] = rng.choice([1, 1, 1, 2, 3, 8]) if cells <= 96 ** 3 else 1
        c["mode"] = rng.choice(["strang", "strang", "strang", "reference_loop", "lie"])
        c["phase"] = rng.choice(["precise", "precise", "precise", "plain"])
        c["grid"] = rng.choice(["periodic", "periodic", "reference"])
        c["tide"] = rng.random() < 0.5
        if c["tide"] and not graph:
            c["centre"] = rng.choice(["box_centre", "box_centre", "reference", "density_max"])
        if c["batch"] == 1 and rng.random() < 0.4:
            c["baryons"] = int(math.exp(rng.uniform(math.log(100), math.log(100_000))))
        c["kerr"] = rng.choice([0.0, 0.0, round(rng.uniform(-0.5, 0.5), 3)])
        c["absorb"] = rng.choice([0.0, 0.0, round(rng.uniform(0.5, 4.0), 2)])
        c["potential"] = rng.random() < 0.2
        return c
    if kind == "ensemble":
        sizes = sorted(rng.sample([16, 24, 32, 48, 64, 96, 128], rng.randint(1, 3)))
        most = 40_000_000 // len(sizes)
        groups = ",".join("%d:%d" % (s, max(1, min(128, int(most / s ** 3 * math.exp(-rng.uniform(0, 4)))))) for s in sizes)
        return dict(kind=kind, groups=groups, steps=rng.randint(1, 10), box=box)
    if kind == "adjoint":
        return dict(kind=kind, steps=rng.randint(3, 40), every=rng.randint(1, 12), box=box,
                    **_draw_axes(rng, 14, 128, 128 ** 3))
    if kind == "snapshot":
        return dict(kind=kind, box=box, **_draw_axes(rng, 10, 300, 256 ** 3))
    if kind == "poisson":
        return dict(kind=kind, box=box, **_draw_axes(rng, 10, 500, 512 ** 3))
    if kind == "fft":
        return dict(kind=kind, inverse=rng.random() < 0.5, **_draw_axes(rng, 10, 500, 512 ** 3))
    if kind == "solver":
        return dict(kind=kind, steps=rng.randint(5, 40), every=rng.randint(3, 12), box=box, **_draw_axes(rng, 14, 80, 64 ** 3))
    if kind == "host":
        return dict(kind=kind, box=box, **_draw_axes(rng, 14, 280, 256 ** 3))
    return dict(kind=kind, steps=rng.randint(1, 8), box=box, **_draw_axes(rng, 14, 280, 256 ** 3))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    """Points and box lengths per axis (x, y, z): spacings are equal, the longest edge is `box`."""
    n = (case["nx"], case["ny"], case["nz"])
    d = case["box"] / max(n)
    return n, tuple(d * k for k in n)


def _dt(case):
    n, _ = _shape(case)
    return (case["box"] / max(n)) ** 2 / 6.0


def _axes(n, L, grid):
    """Coordinates and wavenumbers per axis, FP64, shaped to broadcast over [z][y][x]."""
    x, k = [], []
    for a in range(3):
        s = [1, 1, 1]
        s[2 - a] = n[a]
        d = L[a] / (n[a] - 1 if grid == "reference" else n[a])
        x.append((-L[a] / 2 + d * torch.arange(n[a], dtype=torch.float64, device=DEV)).reshape(s))
        k.append((2 * math.pi * torch.fft.fftfreq(n[a], 1.0 / n[a], dtype=torch.float64, device=DEV) / L[a]).reshape(s))
    return x, k


def _halo(n, L, g, grid="periodic"):
    """A moving soliton off the centre plus a random-phase halo under an NFW-like envelope (complex64 [z][y][x])."""
    x, k = _axes(n, L, grid)
    u = torch.rand(8, generator=g, device=DEV, dtype=torch.float64)
    off = [(float(u[a]) - 0.5) * 0.2 * L[a] for a in range(3)]
    r2 = sum((x[a] - off[a]) ** 2 for a in range(3)).float()
    w = torch.complex(*(torch.randn(n[::-1], generator=g, device=DEV) for _ in "ri"))
    w = torch.fft.ifftn(w * torch.exp(-sum(q * q for q in k) / 4.0).float())
    w = w / w.abs().square().mean().sqrt()
    r = (r2.sqrt() + L[0] / n[0]) / 4.0
    env = 1.0 / (r * (1 + r) ** 2)
    rc = 0.8 + 1.2 * float(u[3])
    move = sum(2 * math.pi / L[a] * x[a] for a in range(3)).float()  # one lattice wavenumber per axis
    core = torch.polar((1.0 + 0.091 * r2 / rc ** 2) ** -4, move.expand(r2.shape).contiguous())
    return (core + (env * (0.01 / env.mean())).sqrt() * w).to(torch.complex64).contiguous()


def _tide_rows(case, g):
    """A host's tidal tensor along an orbit: rows (xx, yy, zz, xy, xz, yz) at s dt."""
    a = 0.01 * (0.5 + float(torch.rand(1, generator=g, device=DEV)))
    rows = []
    for s in range(case["steps"] + 1):
        c, q = math.cos(0.05 * s), math.sin(0.05 * s)
        rows.append([a * (2 * c * c - q * q), a * (2 * q * q - c * c), -a, a * 3 * c * q, 0.1 * a, -0.05 * a])
    return np.array(rows[:1] if case["graph"] or case["batch"] > 1 else rows)


def _stars(case, L, g):
    """A Plummer sphere of static particles, inside the box."""
    m = case["baryons"]
    u, c, f = (torch.rand(m, generator=g, device=DEV, dtype=torch.float64) for _ in "ucf")
    r = (0.5 / torch.sqrt((0.02 + 0.95 * u) ** (-2.0 / 3.0) - 1.0)).clamp(max=0.4 * min(L))
    z = 2 * c - 1
    s = (1 - z * z).sqrt()
    pos = torch.stack([r * s * torch.cos(2 * math.pi * f), r * s * torch.sin(2 * math.pi * f), r * z], 1)
    return pos.cpu().numpy(), np.full(m, 10.0 / m)


def _gen(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _inputs(case, seed):
    """Everything a case is given, on the GPU or (host programs) the host; the same for prepare() and exact()."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "fft":
        n = (case["nx"], case["ny"], case["nz"])
        return dict(data=torch.complex(*(torch.randn(n[::-1], generator=g, device=DEV) for _ in "ri")))
    if kind == "ensemble":
        out = []
        for part in case["groups"].split(","):
            n, b = (int(v) for v in part.split(":"))
            L = (case["box"],) * 3
            psi = torch.empty((b, n, n, n), dtype=torch.complex64, device=DEV)
            for i in range(b):
                psi[i] = _halo((n,) * 3, L, g)
            a = 0.05 * torch.rand(b, generator=g, device=DEV, dtype=torch.float64).cpu().numpy()
            out.append(dict(n=n, batch=b, L=L, psi=psi if b > 1 else psi[0], dt=(case["box"] / n) ** 2 / 6.0,
                            tide=np.stack([2 * a, -a, -a, 0 * a, 0 * a, 0 * a], 1)))
        return out
    n, L = _shape(case)
    if kind == "poisson":
        return dict(rho=_halo(n, L, g).abs().square())
    got = dict(psi=_halo(n, L, g, case.get("grid", "periodic")))
    if kind == "step":
        if case["batch"] > 1:
            got["psi"] = torch.stack([got["psi"]] + [_halo(n, L, g, case["grid"]) for _ in range(case["batch"] - 1)])
        if case["tide"]:
            got["tide"] = _tide_rows(case, g)
        if case["baryons"]:
            got["stars"] = _stars(case, L, g)
        if case["potential"]:  # a shallow trap
            x, _ = _axes(n, L, case["grid"])
            v = sum(0.005 * (x[a] - 0.1 * L[a]) ** 2 for a in range(3)).float()
            got["V"] = v if case["batch"] == 1 else v.expand(got["psi"].shape).contiguous()
    if kind == "adjoint":
        got["target"] = _halo(n, L, g).abs().square()
        got["amp"] = torch.tensor(0.02, dtype=torch.float64)
    if kind in ("solver", "host"):
        got["psi"] = got["psi"].cpu()
        if kind == "host":
            got["psi"] = got["psi"].pin_memory()
    return got


TIDE_DIRECTION = (2.0, -1.0, -1.0, 0.5, 0.0, 0.0)


def prepare(case, seed):
    s = dict(case=case, inp=_inputs(case, seed))
    kind, inp = case["kind"], s["inp"]
    if kind == "ensemble":
        s["members"] = [wdm.SPEContext((m["n"],) * 3, m["L"], batch=m["batch"]) for m in inp]
        for c, m in zip(s["members"], inp):
            c.set_tidal(m["tide"], per_item=True)
        s["group"] = wdm.Ensemble(s["members"])
        s["dts"] = [m["dt"] for m in inp]
        s["out"] = [torch.empty_like(m["psi"]) for m in inp]
        return s
    if kind == "fft":
        n = (case["nx"], case["ny"], case["nz"])
        s["ctx"] = wdm.SPEContext(n, (1.0, 1.0, 1.0))
        s["out"] = torch.empty_like(inp["data"])
        return s
    n, L = _shape(case)
    s["dt"] = _dt(case)
    if kind == "solver":
        return s
    if kind == "step":
        c = wdm.SPEContext(n, L, convention=case["grid"], kerr=case["kerr"], absorb_alpha=case["absorb"],
                           phase_mode=case["phase"], batch=case["batch"])
        if case["tide"]:
            if len(inp["tide"]) > 1:
                c.set_tidal(inp["tide"], t_first=0.0, t_step=s["dt"])
            else:
                c.set_tidal(inp["tide"])
            c.set_tidal_centering(case["centre"])
        if case["baryons"]:
            c.set_particles(*inp["stars"])
        if case["potential"]:
            c.set_static_potential(inp["V"])
    else:
        c = wdm.SPEContext(n, L)
    s["ctx"] = c
    if kind == "poisson":
        s["out"] = torch.empty_like(inp["rho"])
    elif kind == "host":
        s["in"] = inp["psi"].numpy()
        s["out"] = torch.empty_like(inp["psi"]).pin_memory().numpy()
    elif kind == "snapshot":
        s["rho"] = torch.empty(inp["psi"].shape, device=DEV)
        s["phi"] = torch.empty(inp["psi"].shape, device=DEV)
    elif kind == "adjoint":
        inp["psi"].requires_grad_(True)
        inp["amp"].requires_grad_(True)
    else:
        s["out"] = torch.empty_like(inp["psi"])
    return s


def run(s):
    case, inp = s["case"], s["inp"]
    kind = case["kind"]
    if kind == "ensemble":
        for c, m in zip(s["members"], inp):
            c.set_psi(m["psi"])
        s["group"].step(case["steps"], s["dts"])
        return [c.get_psi(o) for c, o in zip(s["members"], s["out"])]
    if kind == "fft":
        s["out"].copy_(inp["data"])
        torch.cuda.current_stream().synchronize()  # the transform runs on the context's own stream
        return s["ctx"].fft3d(s["out"], inverse=case["inverse"])
    if kind == "poisson":
        return s["ctx"].poisson(inp["rho"], s["out"])
    if kind == "solver":
        n, L = _shape(case)
        got = solver.SPE3D_waveDM(Nx=n[0], Ny=n[1], Nz=n[2], Xmax=L[0] / 2, Ymax=L[1] / 2, Zmax=L[2] / 2,
                                  Nt=case["steps"] + 1, Tmax=float(np.float32(s["dt"])) * (case["steps"] + 1), IC=inp["psi"].numpy(),
                                  StepsBetweenSnapshots=case["every"], keep_snapshots=True, poisson_coeff=1.0)
        return [got["psi"]] + got["snapshots"]
    c = s["ctx"]
    if kind == "host":
        c.set_psi(s["in"])
        c.step(1, s["dt"])
        return c.get_psi(s["out"])
    if kind == "adjoint":
        inp["psi"].grad = inp["amp"].grad = None
        loss = autograd.evolve_loss(inp["psi"], inp["amp"], c, case["steps"], s["dt"], inp["target"], TIDE_DIRECTION,
                                    ckpt_every=case["every"])
        loss.backward()
        # the two numbers are sums over an FP32 state
        return [loss.detach().float(), inp["psi"].grad, inp["amp"].grad.float()]
    c.set_psi(inp["psi"])
    if kind == "snapshot":
        return [c.diagnostics(), c.get_rho(s["rho"]), c.get_phi(s["phi"])]
    if kind == "operators":
        for i in range(case["steps"]):
            solver.apply_kick_step(c, s["dt"] / 2, t=i * s["dt"])
            solver.apply_drift_step(c, s["dt"])
    elif case["graph"]:
        c.step_graph(case["steps"], s["dt"], mode=case["mode"])
    else:
        c.step(case["steps"], s["dt"], mode=case["mode"])
    return c.get_psi(s["out"])


# ---------------------------------------------------------------------------
# the least a pass has to move and compute
# ---------------------------------------------------------------------------
def _step_flops(n, logn):
    # two complex transforms, two real ones, phases, density and the two multiplications in k space
    return n * (2 * 5 * logn + 2 * 2.5 * logn + 60)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        n = [(int(a) ** 3 * int(b), 3 * math.log2(int(a))) for a, b in (p.split(":") for p in case["groups"].split(","))]
        return dict(bytes=sum(16 * c for c, _ in n), flops=case["steps"] * sum(_step_flops(c, l) for c, l in n))
    cells = case["nx"] * case["ny"] * case["nz"]
    logn = math.log2(cells)
    if kind == "fft":
        return dict(bytes=16 * cells, flops=5 * cells * logn)
    if kind == "poisson":
        return dict(bytes=8 * cells, flops=5 * cells * logn + 5 * cells)
    if kind == "snapshot":
        return dict(bytes=16 * cells, flops=5 * cells * logn + 80 * cells)
    if kind == "adjoint":
        return dict(bytes=20 * cells, flops=2.5 * case["steps"] * _step_flops(cells, logn))
    if kind == "solver":
        return dict(bytes=8 * cells * (2 + -(-case["steps"] // case["every"])), flops=case["steps"] * _step_flops(cells, logn))
    if kind == "host":
        return dict(bytes=16 * cells, flops=_step_flops(cells, logn))
    cells *= case.get("batch", 1)
    return dict(bytes=16 * cells + (4 * cells if case.get("potential") else 0), flops=case["steps"] * _step_flops(cells, logn))


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
class _Box:
    def __init__(self, n, L, grid="periodic"):
        self.n, self.L = n, L
        self.x, self.k = _axes(n, L, grid)
        self.d = [L[a] / (n[a] - 1 if grid == "reference" else n[a]) for a in range(3)]
        self.k2 = sum(q * q for q in self.k)
        h = self.k2[..., : n[0] // 2 + 1].clone()
        h[0, 0, 0] = 1.0
        self.green = -1.0 / h
        self.green[0, 0, 0] = 0.0

    def poisson(self, rho):
        return torch.fft.irfftn(torch.fft.rfftn(rho) * self.green, s=rho.shape)

    def tide(self, T, x=None):
        x = x or self.x
        xx, yy, zz, xy, xz, yz = T
        return (0.5 * (xx * x[0] ** 2 + yy * x[1] ** 2 + zz * x[2] ** 2) + xy * x[0] * x[1] + xz * x[0] * x[2]
                + yz * x[1] * x[2])

    def centred_tide(self, T, rho, centre):
        if centre == "box_centre":
            return self.tide(T)
        c = np.unravel_index(int(torch.argmax(rho)), tuple(rho.shape))
        xc = [float(self.x[a].reshape(-1)[int(c[2 - a])]) for a in range(3)]
        xx, yy, zz, xy, xz, yz = T
        grad = [xx * xc[0] + xy * xc[1] + xz * xc[2], xy * xc[0] + yy * xc[1] + yz * xc[2],
                xz * xc[0] + yz * xc[1] + zz * xc[2]]
        if centre == "reference":
            return self.tide(T) - 0.5 * sum(p * q for p, q in zip(grad, xc))
        mean = [float((self.x[a] * rho).sum() / rho.sum()) for a in range(3)]
        return (self.tide(T, [self.x[a] - xc[a] for a in range(3)])
                + sum(grad[a] * (mean[a] - xc[a]) for a in range(3)))

    def mask(self, alpha, dt):
        s = 0.0
        for a in range(3):
            X, w = self.L[a] / 2, self.L[a] / 100
            s = s + 2.0 - torch.tanh((self.x[a] + X) / w) + torch.tanh((self.x[a] - X) / w)
        return torch.exp(-alpha * dt * s)

    def cic(self, pos, mass):
        i, f = [], []
        for a in range(3):
            u = (torch.as_tensor(pos[:, a], device=DEV) + self.L[a] / 2) / self.d[a]
            i.append(torch.floor(u).long())
            f.append(u - torch.floor(u))
        rho = torch.zeros(self.n[0] * self.n[1] * self.n[2], dtype=torch.float64, device=DEV)
        m = torch.as_tensor(mass, device=DEV) / (self.d[0] * self.d[1] * self.d[2])
        for corner in range(8):
            o = [(corner >> a) & 1 for a in range(3)]
            w = m
            for a in range(3):
                w = w * (f[a] if o[a] else 1 - f[a])
            j = [(i[a] + o[a]) % self.n[a] for a in range(3)]
            rho.index_add_(0, (j[2] * self.n[1] + j[1]) * self.n[0] + j[0], w)
        return rho.reshape(self.n[::-1])

    def evolve(self, psi, steps, dt, mode="strang", kerr=0.0, absorb=0.0, V=None, rho_b=None, tide=None,
               centre="box_centre", keep=None):
        mask = self.mask(absorb, dt) if absorb else None
        drift = torch.polar(torch.ones_like(self.k2), -0.5 * dt * self.k2)

        def kick(p, h, s):
            rho = p.real.square() + p.imag.square()
            pot = self.poisson(rho if rho_b is None else rho + rho_b)
            if kerr:
                pot = pot + kerr * rho
            if V is not None:
                pot = pot + V
            if tide is not None:
                pot = pot + self.centred_tide(tide[min(s, len(tide) - 1)], rho, centre)
            return p * torch.exp(-1j * h * pot)

        for s in range(steps):
            psi = kick(psi, dt if mode == "lie" else dt / 2, s)
            psi = torch.fft.ifftn(torch.fft.fftn(psi) * drift)
            if mask is not None:
                psi = psi * mask
            if mode == "strang":
                psi = kick(psi, dt / 2, s + 1)
            if keep is not None:
                keep(s + 1, psi)
        return psi

    def record(self, psi, phi):
        """Diagnostics of the reference's loop (its central differences and sums run over interior cells)."""
        dV = self.d[0] * self.d[1] * self.d[2]
        rho = psi.real.square() + psi.imag.square()
        mass = rho.sum()
        top = int(torch.argmax(rho))
        inner = (slice(1, -1),) * 3

        def grad(f, a):
            lo, hi = [slice(1, -1)] * 3, [slice(1, -1)] * 3
            lo[2 - a], hi[2 - a] = slice(None, -2), slice(2, None)
            return (f[tuple(hi)] - f[tuple(lo)]) / (2 * self.d[a])

        c, ri = psi[inner].conj(), rho[inner]
        j = [(c * grad(psi, a)).imag for a in range(3)]
        W = float(-0.5 * (ri * phi[inner]).sum() * dV)
        K = float(0.5 * (sum(q * q for q in j) / ri).nan_to_num(0.0).sum() * dV)
        size = rho.sqrt()
        Q = float(0.5 * sum(grad(size, a).square() for a in range(3)).sum() * dV)
        z = max(self.n[2] // 2 - 1, 0)
        w = rho[z]
        r = (self.x[0][0] ** 2 + self.x[1][0] ** 2 + self.x[2][z] ** 2).sqrt()
        mean = (w * r).sum() / w.sum()
        rmax, pmax = float(rho.reshape(-1)[top]), float(phi.abs().max())
        rec = dict(mass=float(mass) * dV, rho_max=rmax, argmax=float(top), VirialPotential=W, TotalKineticE=K,
                   TotalQuantumE=Q, Virial=2 * K + 2 * Q - W, phi_abs_max=pmax, psi_abs_max=math.sqrt(rmax),
                   dt_phase=2 * self.d[0] ** 2 / math.pi, dt_grav=2 * math.pi / pmax, dt_self=math.inf,
                   R=math.sqrt(max(0.0, float((w * r * r).sum() / w.sum() - mean * mean))))
        for a, name in enumerate("xyz"):
            rec["com_" + name] = float((rho * self.x[a]).sum() / mass)
            rec["Momentum" + name.upper()] = float(j[a].sum() * dV)
        # weighted quantiles of the distance from the densest cell, by its square in cells
        at = np.unravel_index(top, tuple(rho.shape))
        key = 0
        for a in range(3):
            s = [1, 1, 1]
            s[2 - a] = self.n[a]
            key = key + ((torch.arange(self.n[a], device=DEV) - int(at[2 - a])) ** 2).reshape(s)
        wsum = torch.bincount(key.reshape(-1), weights=rho.reshape(-1)).cpu().numpy()
        group = np.flatnonzero(wsum > 0)
        cum = np.cumsum(wsum[group])
        for q in range(1, 10):
            h = 0.1 * q * (cum[-1] - rmax) + rmax
            k = int(np.searchsorted(cum, h, side="right"))
            if k >= len(group):
                rec["radius_%d0" % q] = self.d[0] * math.sqrt(group[-1])
                continue
            value = math.sqrt(group[k])
            before, last = (cum[k - 1], math.sqrt(group[k - 1])) if k else (0.0, 0.0)
            least = float(rho[(key == int(group[k])) & (rho > 0)].min())
            if h < before + least:
                value = last + (h - before) / least * (value - last)
            rec["radius_%d0" % q] = self.d[0] * value
        return rec


def exact(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m in inp:
            box = _Box((m["n"],) * 3, m["L"])
            psi = m["psi"] if m["batch"] > 1 else m["psi"][None]
            got = torch.stack([box.evolve(p.to(torch.complex128), case["steps"], m["dt"], tide=[T])
                               for p, T in zip(psi, m["tide"])])
            out.append(got if m["batch"] > 1 else got[0])
        return out
    if kind == "fft":
        data = inp["data"].to(torch.complex128)
        return torch.fft.ifftn(data, norm="forward") if case["inverse"] else torch.fft.fftn(data)
    n, L = _shape(case)
    dt = _dt(case)
    if kind == "poisson":
        return _Box(n, L).poisson(inp["rho"].double())
    if kind == "solver":
        kept = []

        def keep(s, psi):
            if s % case["every"] == 0 or s == case["steps"]:
                kept.append(psi.clone())

        dt = float(np.float32(dt))  # the solver's time step is FP32, as the reference's
        psi = _Box(n, L, "reference").evolve(inp["psi"].to(DEV, torch.complex128), case["steps"], dt,
                                             mode="reference_loop", keep=keep)
        return [psi] + kept
    if kind == "host":
        return _Box(n, L).evolve(inp["psi"].to(DEV, torch.complex128), 1, dt)
    psi = inp["psi"].to(torch.complex128)
    if kind == "adjoint":
        box = _Box(n, L)
        psi.requires_grad_(True)
        amp = inp["amp"].to(DEV).requires_grad_(True)
        end = box.evolve(psi, case["steps"], dt, tide=[[amp * d for d in TIDE_DIRECTION]])
        diff = end.real.square() + end.imag.square() - inp["target"].double()
        loss = diff.square().sum() * box.d[0] * box.d[1] * box.d[2]
        loss.backward()
        return [loss.detach(), psi.grad, amp.grad]
    if kind == "snapshot":
        box = _Box(n, L)
        rho = psi.real.square() + psi.imag.square()
        phi = box.poisson(rho)
        return [box.record(psi, phi), rho, phi]
    if kind == "operators":
        return _Box(n, L).evolve(psi, case["steps"], dt, mode="reference_loop")
    box = _Box(n, L, case["grid"])
    rho_b = box.cic(*inp["stars"]) if case["baryons"] else None
    V = inp["V"].double() if case["potential"] else None
    items = []
    for i, p in enumerate(psi if case["batch"] > 1 else psi[None]):
        v = None if V is None else V[i] if case["batch"] > 1 else V
        items.append(box.evolve(p, case["steps"], dt, mode=case["mode"], kerr=case["kerr"], absorb=case["absorb"],
                                V=v, rho_b=rho_b, tide=inp.get("tide"), centre=case["centre"]))
    return torch.stack(items) if case["batch"] > 1 else items[0]
