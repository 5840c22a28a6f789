"""Workloads of the library, one dict each, run through its public entry points.

A pass advances a simulation by a number of lattice steps (or trains the pair
closure) and hands the result to the caller: the populations as a packed device
snapshot (lbx_pack_planes, stored form), the moments as host arrays
(LBSim.get_fields), the sphere records (LBSim.get_particles) or the trained
weights.  `exact` states the fluid models and the training in 64 bits with plain
torch.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from lbcuda_b200 import LBSim, capi, closure, make_params
from lbcuda_b200.ensemble import Ensemble, random_boxes

SIGMA, BETA = 0.02, 0.7
HALF_TYPES = {"f16": torch.float16, "f16sd": torch.float16, "f16sdp": torch.float16,
              "bf16": torch.bfloat16, "bf16sd": torch.bfloat16, "bf16sdp": torch.bfloat16}
DENS_R = 2.0  # red density of the two-density model (the namelist deck of the reference)


def listed():
    return [
        # plain BGK in a small periodic box, the first configuration: latency and cache
        dict(name="bgk_64_f32", kind="fluid", model="bgk", storage="f32", nx=64, ny=64, nz=64, steps=100,
             field="noise"),
        # a small colour-gradient box advanced a few steps per call: launches and latency
        dict(name="spinodal_32_f32", kind="fluid", model="cg", storage="f32", nx=32, ny=32, nz=32, steps=10,
             field="noise"),
        # the colour-gradient workload in the reference's own storage type
        dict(name="spinodal_128_f32", kind="fluid", model="cg", storage="f32", nx=128, ny=128, nz=128, steps=20,
             field="noise"),
        # the benchmark's storage, with an output interval: steps, then moments on the host
        dict(name="output_128_f16sd", kind="fluid", model="cg", storage="f16sd", nx=128, ny=128, nz=128, steps=100,
             field="noise", fields=True),
        # the same at a box that streams from HBM
        dict(name="spinodal_256_f16sd", kind="fluid", model="cg", storage="f16sd", nx=256, ny=256, nz=256, steps=20,
             field="noise"),
        # a droplet in a flow: an odd box, two viscosities, the storage with the smallest error
        dict(name="droplet_odd_f16sdp", kind="fluid", model="cg", storage="f16sdp", nx=150, ny=97, nz=75, steps=20,
             field="droplet", tauB=0.8),
        # two fluid densities (the reference's namelist deck)
        dict(name="diffdens_128_f32", kind="fluid", model="cg-diffdens", storage="f32", nx=128, ny=128, nz=128,
             steps=20, field="droplet"),
        # the D3Q27 lattice
        dict(name="d3q27_96_f32", kind="fluid", model="cg-d3q27", storage="f32", nx=96, ny=96, nz=96, steps=20,
             field="noise"),
        # 1280 spheres in 256^3: the suspension workload
        dict(name="colloid_256_f16sd", kind="colloid", storage="f16sd", nx=256, ny=256, nz=256, steps=20,
             spheres=1280, wetting="neutral"),
        # a few spheres in a small box: the sphere kernels' latency, FP32, Janus wetting
        dict(name="colloid_48_f32", kind="colloid", storage="f32", nx=48, ny=48, nz=48, steps=20, spheres=8,
             wetting="janus"),
        # 48 uneven boxes with spheres and the closure advanced together, tuned
        dict(name="ensemble_48_f16sd", kind="ensemble", storage="f16sd", boxes=48, steps=20),
        # training of the pair closure: the data of all 121 lattice classes, two epochs
        dict(name="closure_train", kind="train", n=30976, epochs=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fluid", "fluid", "fluid", "fluid", "colloid", "colloid", "train", "ensemble"])
    if kind == "train":
        return dict(kind="train", n=_log_int(rng, 500, 30000), epochs=rng.randint(1, 3))
    if kind == "ensemble":
        return dict(kind="ensemble", storage=rng.choice(["f16sd", "f32"]), boxes=rng.randint(2, 24),
                    steps=rng.randint(4, 20))
    if kind == "colloid":
        nx, ny, nz = (_log_int(rng, 5, 20) * 8, _log_int(rng, 10, 40) * 4, _log_int(rng, 10, 40) * 4)
        return dict(kind="colloid", storage=rng.choice(["f32", "f16sd", "f16"]), nx=nx, ny=ny, nz=nz,
                    steps=rng.randint(5, 20), spheres=rng.randint(1, max(1, nx * ny * nz // 16000)),
                    wetting=rng.choice(["janus", "neutral"]))
    model = rng.choice(["bgk", "cg", "cg", "cg", "cg-diffdens", "cg-d3q27"])
    storage = rng.choice(["f32", "f16", "f16sd", "f16sdp", "bf16sd"]) if model == "cg" else "f32"
    dims = [_log_int(rng, 20, 200) for _ in range(3)]
    if rng.random() < 0.5:  # common boxes: x a multiple of 16
        dims[0] = max(16, dims[0] // 16 * 16)
    case = dict(kind="fluid", model=model, storage=storage, nx=dims[0], ny=dims[1], nz=dims[2],
                steps=rng.randint(2, 20), field="droplet" if model == "cg-diffdens" else rng.choice(["noise", "droplet"]))
    if model in ("cg", "cg-diffdens") and rng.random() < 0.3:
        case["tauB"] = round(rng.uniform(0.7, 1.3), 3)
    return case


# ---- inputs -----------------------------------------------------------------
def _gen(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fields(case, seed):
    """(rhoR, rhoB, velocity) as float32 host arrays; rhoB is None for one component."""
    dev = _device()
    g = _gen(seed, dev)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]

    def noise(amp):
        return (torch.rand((nz, ny, nx), generator=g, device=dev) * 2 - 1) * amp

    if case.get("model") == "bgk":
        return (1.0 + noise(1e-3)).float().cpu().numpy(), None, (0.0, 0.0, 0.0)
    if case.get("field", "noise") == "noise":
        return (0.5 + noise(0.01)).float().cpu().numpy(), (0.5 + noise(0.01)).float().cpu().numpy(), (0.0, 0.0, 0.0)
    # droplet of an eighth of the shortest edge near the centre, an interface
    # of about a cell, in a uniform flow, a little density noise on both sides
    at = torch.rand(4, generator=g, device=dev).tolist()
    k, j, i = torch.meshgrid(*[torch.arange(n, device=dev, dtype=torch.float32) for n in (nz, ny, nx)], indexing="ij")
    r = min(nx, ny, nz) / 8.0 + at[3]
    d = torch.sqrt((i - nx / 2 - at[0]) ** 2 + (j - ny / 2 - at[1]) ** 2 + (k - nz / 2 - at[2]) ** 2)
    t = torch.clamp(0.5 - (d - r) / 2.0, 0.0, 1.0)
    scale = DENS_R if case["model"] == "cg-diffdens" else 1.0
    return ((t * scale * (1.0 + noise(1e-3))).float().cpu().numpy(),
            ((1.0 - t) * (1.0 + noise(1e-3))).float().cpu().numpy(), (0.02, 0.01, 0.005))


def _spheres(rng, n, box, dist):
    """n centres in [1, L] with periodic distances of at least `dist` (fewer if the box fills up)."""
    L = np.array(box, np.float64)
    x = np.empty((0, 3))
    for _ in range(400 * n):
        if len(x) == n:
            break
        c = rng.uniform(1.0, L)
        d = x - c
        d -= L * np.round(d / L)
        if not len(x) or (d * d).sum(1).min() >= dist * dist:
            x = np.vstack([x, c])
    return x


def _fluid_params(case, **more):
    extra = {"tauB": case["tauB"]} if "tauB" in case else {}
    if case.get("model") == "cg-diffdens":
        extra.update(densR=DENS_R, densB=1.0)
    return make_params(case["nx"], case["ny"], case["nz"], model=case.get("model", "cg"), storage=case["storage"],
                       sigma=SIGMA, beta=BETA, **extra, **more)


class Snapshot:
    """A device buffer for the packed populations of a context (the caller's, kept between passes)."""

    def __init__(self, sim, storage):
        n = ctypes.c_int64()
        capi.check(capi.lib().lbx_plane_bytes(sim._h, sim.nz, ctypes.byref(n)))
        self.sim, self.buf = sim, torch.empty(n.value, dtype=torch.uint8, device=_device())
        cells = sim.nx * sim.ny * sim.nz
        dt = HALF_TYPES.get(storage, torch.float32)
        q = getattr(sim, "q", 19)  # an ensemble's boxes are D3Q19
        width = q * cells * sim.ncomp * (2 if storage in HALF_TYPES else 4)
        self.out = {"pops": self.buf[:width].view(dt).view(q, sim.nz, sim.ny, sim.nx, sim.ncomp)}
        if width < n.value:  # predicted split: the phase field the pairs are encoded against
            self.out["split"] = self.buf[width:].view(torch.float32).view(sim.nz, sim.ny, sim.nx)

    def take(self):
        capi.check(capi.lib().lbx_pack_planes(self.sim._h, 0, self.sim.nz, self.buf.data_ptr()), "lbx_pack_planes")
        return self.out


def _train_data(case, seed):
    """Features and targets of sphere pairs: gaps log-uniform, pair-frame velocities uniform in +-1e-3, lattice
    directions; a squeeze and shear resistance of the gap as the targets."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    gap = np.exp(rng.uniform(np.log(0.05), np.log(1.5), n))
    q = rng.uniform(-1e-3, 1e-3, (n, 9))
    nc = -np.sort(-np.abs(rng.normal(size=(n, 3))), axis=1)
    nc /= np.linalg.norm(nc, axis=1, keepdims=True)
    X = np.concatenate([gap[:, None], q, np.full((n, 1), 3.0), nc[:, 1:3]], axis=1)
    M = rng.normal(size=(9, 12)) * 0.3
    squeeze, shear = 1.0 / gap, np.log(1.0 + 1.0 / gap)
    T = (q @ M) * (shear * (1.0 + nc[:, 1]))[:, None]
    T[:, 0] += q[:, 0] * squeeze
    T[:, 6] -= q[:, 0] * squeeze
    return X.astype(np.float32), T.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, T = _train_data(case, seed)
        return dict(case=case, X=X, T=T, seed=seed & 0xffff)
    if kind == "ensemble":
        return _prepare_ensemble(case, seed)
    if kind == "fluid":
        sim = LBSim(_fluid_params(case))
        rR, rB, vel = _fields(case, seed)
        sim.set_fields(rR, rB, vel)
        return dict(case=case, sim=sim, snap=None if case.get("fields") else Snapshot(sim, case["storage"]))
    rng = np.random.default_rng(seed)
    x = _spheres(rng, case["spheres"], (case["nx"], case["ny"], case["nz"]), 13.0)
    sim = LBSim(_fluid_params(case, max_particles=len(x), radius=5.5, rmass=1.0 / (4.0 / 3.0 * math.pi * 5.5 ** 3),
                              wetting=case["wetting"], lrotate=1, max_vel=1.0))
    rR, rB, vel = _fields(case, seed)
    sim.set_fields(rR, rB, vel)
    sim.set_particles(x, rng.uniform(-0.01, 0.01, x.shape))
    return dict(case=case, sim=sim, snap=Snapshot(sim, case["storage"]))


def _prepare_ensemble(case, seed):
    # the boxes themselves stay those of the workload (seed 7); the fields and velocities come from the seed
    spec = _boxes(case["boxes"])
    params = [make_params(L, model="cg", storage=case["storage"], sigma=SIGMA, beta=BETA, max_particles=max(len(x), 1),
                          radius=4.0, wetting="neutral", lrotate=1, max_vel=1.0, exact_tiles=0, hz_rmin=8.5,
                          hz_rcap=7.0, closure=1, lubrication=1, lubric_rmin=1.0, lubric_rcap=0.2)
              for L, x in spec]
    ens = Ensemble(params)
    w = np.zeros(closure.NW, np.float32)
    F = ctypes.POINTER(ctypes.c_float)
    capi.check(capi.lib().lbx_closure_init(w.ctypes.data_as(F), 1))
    w[closure.YSD:closure.YSD + closure.DOUT] = 1e-4  # untrained corrections of the size of trained ones

    def load():
        rng = np.random.default_rng(seed)
        for i, (L, x) in enumerate(spec):
            rR, rB, _ = _fields(dict(nx=L, ny=L, nz=L), seed * 64 + i)
            ens.boxes[i].set_fields(rR, rB)
            if len(x):
                ens.boxes[i].set_particles(x, rng.uniform(-0.005, 0.005, x.shape))
                capi.check(capi.lib().lbx_closure_set(ens.boxes[i]._h, w.ctypes.data_as(F)))

    load()
    ens.tune(trial=4)
    load()
    return dict(case=case, ens=ens, snaps=[Snapshot(b, case["storage"]) for b in ens.boxes],
                owners=[b for b, (_, x) in zip(ens.boxes, spec) if len(x)])


@functools.lru_cache(maxsize=None)
def _boxes(n):
    """Edges and sphere centres of the ensemble workload's first n boxes (the same for every seed)."""
    return random_boxes(n, seed=7)


# ---- one pass -----------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "train":
        w, loss = closure.train(state["X"], state["T"], epochs=case["epochs"], lr=2e-3, seed=state["seed"])
        return {"weights": w, "loss": loss}
    if case["kind"] == "ensemble":
        state["ens"].step(case["steps"])
        pops = [s.take()["pops"] for s in state["snaps"]]
        parts = [b.get_particles() for b in state["owners"]]
        out = {"pops_%02d" % i: p for i, p in enumerate(pops)}
        for k in parts[0] if parts else ():
            out[k] = np.concatenate([p[k] for p in parts])
        return out
    sim = state["sim"]
    sim.step(case["steps"])
    if case.get("fields"):
        rhoR, rhoB, vel, phase = sim.get_fields()
        return {"rhoR": rhoR, "rhoB": rhoB, "vel": vel, "phase": phase}
    out = dict(state["snap"].take())
    if case["kind"] == "colloid":
        out.update(sim.get_particles())
    return out


# ---- the work of a pass ---------------------------------------------------------
def _per_cell(model, storage):
    """(bytes, operations) of one cell and step: populations read once and written once."""
    q = 27 if model == "cg-d3q27" else 19
    nc = 1 if model == "bgk" else 2
    size = 2 if storage in HALF_TYPES else 4
    split = 8 if storage.endswith("sdp") else 0  # the predicted split's phase field
    return 2 * q * nc * size + split, q * (12 if model == "bgk" else 28)


def work(case):
    if case["kind"] == "train":
        n = case["n"] * case["epochs"]
        weights = 13 * 64 + 2 * 64 * 64 + 64 * 12
        return {"bytes": n * (13 + 12) * 4, "flops": 6 * weights * n}
    if case["kind"] == "ensemble":
        cells = sum(L ** 3 for L, _ in _boxes(case["boxes"]))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    b, f = _per_cell(case.get("model", "cg"), case["storage"])
    out = 24 * cells if case.get("fields") else 0  # the moments
    return {"bytes": cells * case["steps"] * b + out, "flops": cells * case["steps"] * f}


def tolerance(case):
    if case["kind"] == "train":
        # measured 8e-7 against `exact`; Adam divides small gradients by their size, so
        # another order of the sums shows more in single weights
        return {"rel": 1e-5, "max": 2e-3}
    storage, sphere = case["storage"], case["kind"] != "fluid"
    # About four times the error of the path against `exact`: after 20 steps 7e-6 with
    # FP32 populations, 3e-4 to 7e-4 with FP16 and 2.5e-3 with BF16 ones (stored form,
    # the moments after 100 steps).  Sphere forces and torques are small differences
    # of large sums, and a sphere that crosses a cell's edge a rounding earlier moves
    # a whole cell's mass.
    if storage == "f32":
        return {"rel": 1e-3, "max": 5e-2} if sphere else {"rel": 3e-5, "max": 3e-3}
    rel = 1e-2 if sphere or storage.startswith("bf16") else 3e-3
    return {"rel": rel, "max": 40 * rel}


# ---- the same in 64 bits, plain torch --------------------------------------------
E19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
       (-1, 1, 0), (1, -1, 0), (1, 0, 1), (-1, 0, -1), (-1, 0, 1), (1, 0, -1), (0, 1, 1), (0, -1, -1), (0, -1, 1),
       (0, 1, -1)]
E27 = E19 + [(1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (-1, 1, 1), (1, -1, -1), (1, -1, 1), (-1, 1, -1)]


def _tables(q):
    cls = [sum(abs(c) for c in e) for e in E27[:q]]
    w27 = [8 / 27, 2 / 27, 1 / 54, 1 / 216]
    if q == 27:
        w, b = w27, [-10 / 27, 2 / 27, 1 / 54, 1 / 216]
        phi, varphi = [0, 2 / 19, 1 / 38, 1 / 152], [1, -2 / 19, -1 / 38, -1 / 152]
        psi, xi = [-20 / 9, -2 / 9, 1 / 36, 1 / 36], [0, 1 / 3, 1 / 12, 1 / 48]
    else:
        w, b = [1 / 3, 1 / 18, 1 / 36, 0], [-3 / 13.5, 0.5 / 27, 1 / 27, 0]
        phi, varphi = [0, 1 / 12, 1 / 24, 0], [1, -1 / 12, -1 / 24, 0]
        psi, xi = [-5 / 2, -1 / 6, 1 / 24, 0], [0, 1 / 4, 1 / 8, 0]
    return cls, w, b, [3 * v for v in w27], phi, varphi, psi, xi


def _shift(a, e):
    """a(x - e), periodic."""
    if e == (0, 0, 0):
        return a
    return torch.roll(a, shifts=(e[2], e[1], e[0]), dims=(0, 1, 2))


def _dot(e, v):
    s = 0.0
    for c, a in zip(e, v):
        if c:
            s = s + c * a
    return s


def _gradient(phi, a27):
    """Sum over the 26 neighbours of a27 e phi(x + e)."""
    g = [torch.zeros_like(phi) for _ in range(3)]
    for e in E27[1:]:
        p = a27[sum(abs(c) for c in e)] * _shift(phi, (-e[0], -e[1], -e[2]))
        for d in range(3):
            if e[d]:
                g[d] += e[d] * p
    return g


class _Exact:
    def __init__(self, case, seed):
        f32 = lambda v: float(np.float32(v))  # noqa: E731 - parameters travel as float32
        self.model = case["model"]
        self.dd = self.model == "cg-diffdens"
        self.q = 27 if self.model == "cg-d3q27" else 19
        self.E = E27[:self.q]
        self.cls, self.w, self.b, self.a27, self.phi, self.varphi, self.psi, self.xi = _tables(self.q)
        self.sigma, self.beta = f32(SIGMA), f32(BETA)
        self.vR, self.vB = (1.0 - 0.5) / 3, (f32(case.get("tauB", 1.0)) - 0.5) / 3
        self.dens = (DENS_R, 1.0) if self.dd else (1.0, 1.0)
        aB = self.w[0]
        self.alpha = ((1 / (aB - 1)) * (self.dens[1] / self.dens[0]) + 1, aB)
        rR, rB, vel = _fields(case, seed)
        rho = [torch.from_numpy(r).to(_device()).double() for r in (rR, rB) if r is not None]
        u = [f32(v) for v in vel]
        usq = 1.5 * sum(v * v for v in u)
        # the state holds at x what streaming moves to x + e
        self.A = [[_shift(self.equil(r, _dot(e, u), usq, k, l), (-e[0], -e[1], -e[2])) for l, e in enumerate(self.E)]
                  for k, r in enumerate(rho)]
        self.split = None

    def equil(self, rho, eu, usq, k, l):
        c = self.cls[l]
        if self.dd:
            return rho * (self.phi[c] + self.varphi[c] * self.alpha[k] + self.w[c] * (3 * eu + 4.5 * eu * eu - usq))
        return rho * self.w[c] * (1 + 3 * eu + 4.5 * eu * eu - usq)

    def pulled(self):
        return [[_shift(f, e) for f, e in zip(comp, self.E)] for comp in self.A]

    def velocity(self, f, inv):
        total = [sum(c) for c in zip(*f)] if len(f) > 1 else f[0]
        return [inv * sum(e[d] * t for e, t in zip(self.E, total) if e[d]) for d in range(3)]

    def step(self):
        f = self.pulled()
        if self.model == "bgk":
            rho = sum(f[0])
            u = self.velocity(f, 1 / rho)
            usq = 1.5 * sum(v * v for v in u)
            self.A = [[self.equil(rho, _dot(e, u), usq, 0, l) for l, e in enumerate(self.E)]]  # tau = 1
            return
        r = [torch.clamp(sum(c), min=0.0) for c in f]
        rs, (dR, dB) = r[0] + r[1], self.dens
        ph = (r[0] / dR - r[1] / dB) / (r[0] / dR + r[1] / dB)
        self.split = ph
        visc = 1 / (0.5 * (1 + ph) / self.vR + 0.5 * (1 - ph) / self.vB)
        om = 1 / (3 * visc + 0.5)
        inv = 1 / rs
        u = self.velocity(f, inv)
        usq = 1.5 * sum(v * v for v in u)
        g = _gradient(ph, self.a27)
        grads = [_gradient(x, self.a27) for x in r] if self.dd else None
        psq = sum(v * v for v in g)
        on = psq > 1e-20
        pn = torch.sqrt(torch.where(on, psq, torch.ones_like(psq)))
        ipsq = 1 / (pn * pn)
        ac, coef = 2.25 * om * self.sigma, self.beta * r[0] * r[1] * inv * inv
        new = ([], [])
        for l, e in enumerate(self.E):
            c, eu, ep = self.cls[l], _dot(e, u), _dot(e, g)
            h = []
            for k in range(2):
                eq = self.equil(r[k], eu, usq, k, l)
                if self.dd:
                    uG = sum(a * b for a, b in zip(u, grads[k]))
                    tG = sum(2 * a * b * abs(s) for a, b, s in zip(u, grads[k], e))
                    eq = eq + visc * (self.psi[c] * uG + self.xi[c] * tG)
                h.append(f[k][l] * (1 - om) + eq * om)
            fd = h[0] + h[1] + ac * pn * (self.w[c] * ep * ep * ipsq - self.b[c])
            if self.dd:
                zero = torch.zeros_like(rs)
                feq = sum(self.equil(r[k], zero, zero, k, l) for k in range(2))
            else:
                feq = rs * self.w[c]
            t = coef * ep / (math.sqrt(c) * pn) * feq if c else torch.zeros_like(rs)
            new[0].append(torch.where(on, fd * r[0] * inv + t, h[0]))
            new[1].append(torch.where(on, fd * r[1] * inv - t, h[1]))
        self.A = [list(new[0]), list(new[1])]

    def stored(self, storage):
        if len(self.A) == 1:
            return {"pops": torch.stack(self.A[0]).unsqueeze(-1)}
        out = torch.empty((self.q,) + tuple(self.A[0][0].shape) + (2,), dtype=torch.float64, device=self.A[0][0].device)
        for l, e in enumerate(self.E):
            R, B, w = self.A[0][l], self.A[1][l], self.w[self.cls[l]]
            if storage.endswith("sdp"):
                a, b = R + B - w, R - B - _shift(self.split, (-e[0], -e[1], -e[2])) * (R + B)
            elif storage.endswith("sd"):
                a, b = R + B - w, R - B
            elif storage in HALF_TYPES:
                a, b = R - 0.5 * w, B - 0.5 * w
            else:
                a, b = R, B
            out[l, ..., 0], out[l, ..., 1] = a, b
        return {"pops": out, "split": self.split} if storage.endswith("sdp") else {"pops": out}

    def moments(self):
        f = self.pulled()
        r = [sum(c) for c in f]
        u = self.velocity(f, 1 / (r[0] + r[1]))
        return {"rhoR": r[0], "rhoB": r[1], "vel": torch.stack(u, -1), "phase": (r[0] - r[1]) / (r[0] + r[1])}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] != "fluid":
        return None  # the sphere path has no statement in plain torch here
    x = _Exact(case, seed)
    for _ in range(case["steps"]):
        x.step()
    return x.moments() if case.get("fields") else x.stored(case["storage"])


def _glorot(seed):
    """The initial weights of the closure: xorshift, Glorot-uniform, biases zero."""
    mask, s = (1 << 64) - 1, 0x9E3779B97F4A7C15 ^ (seed & 0xffffffffffffffff)
    mats = []
    for o, k in ((64, 13), (64, 64), (64, 64), (12, 64)):
        lim, v = math.sqrt(6.0 / (k + o)), []
        for _ in range(o * k):
            s ^= (s << 13) & mask
            s ^= s >> 7
            s ^= (s << 17) & mask
            v.append(np.float32((2.0 * ((s >> 11) / 9007199254740992.0) - 1.0) * lim))
        mats += [torch.tensor(np.array(v)).double().view(o, k), torch.zeros(o, dtype=torch.float64)]
    return mats


def _exact_train(case, seed):
    X, T = _train_data(case, seed)
    dev, n, epochs, lr, TB = _device(), case["n"], case["epochs"], float(np.float32(2e-3)), 64
    stats = [X.mean(0), np.maximum(X.std(0), 1e-12), T.mean(0), np.maximum(T.std(0), 1e-12)]
    stats = [torch.from_numpy(v.astype(np.float32)).to(dev).double() for v in stats]
    x = (torch.from_numpy(X).to(dev).double() - stats[0]) / stats[1]
    t = (torch.from_numpy(T).to(dev).double() - stats[2]) / stats[3]
    p = [m.to(dev) for m in _glorot(seed & 0xffff)]
    m1, m2 = [torch.zeros_like(a) for a in p], [torch.zeros_like(a) for a in p]
    nb, step, losses, u32 = (n + TB - 1) // TB, 0, [], 0xffffffff
    b1, b2, eps = float(np.float32(0.9)), float(np.float32(0.999)), float(np.float32(1e-8))
    for ep in range(epochs):
        h = ((seed & 0xffff) * 2654435761 + ep * 40503 + 12345) & u32
        off, stride = h % n, 1 + (h >> 8) % n
        while math.gcd(stride, n) != 1:
            stride = stride % n + 1
        total = torch.zeros((), dtype=torch.float64, device=dev)
        for bi in range(nb):
            cnt = min(TB, n - bi * TB)
            idx = (torch.arange(bi * TB, bi * TB + cnt, device=dev) * stride % n + off) % n
            a, z = [x[idx]], []
            for l in range(4):
                z.append(a[-1] @ p[2 * l].T + p[2 * l + 1])
                a.append(z[-1] * torch.sigmoid(z[-1]) if l < 3 else z[-1])
            d = a[-1] - t[idx]
            total += (d * d).sum()
            d = d * (2.0 / (cnt * 12))
            g = [None] * 8
            for l in (3, 2, 1, 0):
                g[2 * l], g[2 * l + 1] = d.T @ a[l], d.sum(0)
                if l:
                    s = torch.sigmoid(z[l - 1])
                    d = (d @ p[2 * l]) * (s * (1 + z[l - 1] * (1 - s)))
            step += 1
            c1, c2 = 1 - b1 ** step, 1 - b2 ** step
            rate = 0.5 * lr * (1 + math.cos(math.pi * (step - 1) / (epochs * nb)))
            for k in range(8):
                m1[k] = b1 * m1[k] + (1 - b1) * g[k]
                m2[k] = b2 * m2[k] + (1 - b2) * g[k] * g[k]
                p[k] = p[k] - rate * (m1[k] / c1) / (torch.sqrt(m2[k] / c2) + eps)
        losses.append(total / (n * 12))
    return {"weights": torch.cat([a.reshape(-1) for a in p + stats]), "loss": torch.stack(losses)}
