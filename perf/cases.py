"""Performance cases of the lattice-Boltzmann library, through its public calls.

Each case is what a program of a user of this library does between two looks
at its results: it holds a domain (or a batch of samples), advances it by a
stretch of time steps and takes the macroscopic fields (density, velocity,
concentration), or runs one iteration of a gradient-based fit.  `prepare`
makes the porous medium from a seed, creates the domain and sets its initial
state; `run` is one pass; `exact` is the same model in plain 64-bit torch.

All domains work on one CUDA stream, as in a program that orders them with
its own work.  Passes continue the run where the last pass left it, except
where a case says that it starts from rest.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "lbgpu-prime-dev_b200"))

import lbx  # noqa: E402
from lbx.batch import Batch  # noqa: E402

# Directions in the library's exchange order: opposites are adjacent and D2Q9
# is the first nine.
_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (1, 1, 0), (-1, -1, 0),
      (-1, 1, 0), (1, -1, 0), (0, 0, 1), (0, 0, -1), (1, 0, 1), (-1, 0, -1), (-1, 0, 1),
      (1, 0, -1), (0, 1, 1), (0, -1, -1), (0, -1, 1), (0, 1, -1)]
_W2 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
_W3 = [1 / 3] + [1 / 18] * 4 + [1 / 36] * 4 + [1 / 18] * 2 + [1 / 36] * 8


def _opp(a):
    return 0 if a == 0 else (a + 1 if a & 1 else a - 1)


# ---- the cases -----------------------------------------------------------------

def listed():
    """
    flow2d    D2Q9 flow between Zou-He pressure faces past discs (the
              reference's own use): FP64 as shipped.
    solute2d  the same with a solute plume, zero-gradient outlet and a sink.
    flow3d    D3Q19 flow through a sphere pack, driven by a body force:
              permeability runs, FP32 shifted or FP64.
    open3d    D3Q19 flow in an open channel (few solids: the dense layout).
    through3d flow and solute through a pack between pressure planes, with
              the outlet record on: breakthrough runs.
    gradient3d one iteration of a fit: forward from rest with checkpoints,
              then the adjoint, for the force, the relaxation times and the
              inlet profile.
    batch     many independent samples of uneven size, advanced together,
              their fields taken to the host at the end.
    job3d     a whole job from host memory: density uploaded, run from
              rest, fields downloaded.
    """
    return [
        # a small 2D lattice looked at often: latency
        dict(name="flow2d_48x67_f64", kind="flow2d", LX=48, LY=67, real=8, porosity=0.7,
             radius=4, steps=20),
        # the 2D configuration's lattice between two frames
        dict(name="flow2d_256_f64", kind="flow2d", LX=256, LY=256, real=8, porosity=0.6,
             radius=8, steps=1000),
        # a 2D lattice larger than the chip's shared memory holds, ragged
        dict(name="flow2d_701x500_f64", kind="flow2d", LX=701, LY=500, real=8, porosity=0.65,
             radius=9, steps=200),
        # the reference's shipped set-up: 2D, two substances, double
        dict(name="solute2d_300x220_f64", kind="solute2d", LX=300, LY=220, real=8, porosity=0.65,
             radius=7, steps=200),
        # a small sample, as a study of many runs one by one
        dict(name="flow3d_64_f32", kind="flow3d", LX=64, LY=64, LZ=64, real=4, model="shifted",
             porosity=0.5, radius=4, steps=100),
        # the benchmark's lattice
        dict(name="flow3d_256_f32", kind="flow3d", LX=256, LY=256, LZ=256, real=4,
             model="shifted", porosity=0.4, radius=6, steps=100),
        # a large image
        dict(name="flow3d_384x360x320_f32", kind="flow3d", LX=384, LY=360, LZ=320, real=4,
             model="shifted", porosity=0.4, radius=6, steps=40),
        # an open channel, odd extents
        dict(name="open3d_193x161x120_f32", kind="open3d", LX=193, LY=161, LZ=120, real=4,
             model="shifted", steps=60),
        # the flow + solute configuration's lattice
        dict(name="through3d_192x192x384_f32", kind="through3d", LX=192, LY=192, LZ=384, real=4,
             porosity=0.35, radius=5, steps=60),
        # one iteration of a fit
        dict(name="gradient3d_128x112x96_f32", kind="gradient3d", LX=128, LY=112, LZ=96, real=4,
             porosity=0.45, radius=4, steps=100, every=25),
        # a study over samples of uneven size
        dict(name="batch_24_f32", kind="batch", samples=24, low=32, high=96, real=4, steps=1000),
        # a whole double-precision job of a ragged image
        dict(name="job3d_150x131x117_f64", kind="job3d", LX=150, LY=131, LZ=117, real=8,
             model="plain", porosity=0.45, radius=5, steps=200),
    ]


def _between(rng, lo, hi):
    """Log-uniform integer."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow2d", "flow2d", "solute2d", "flow3d", "flow3d", "flow3d", "open3d",
                       "through3d", "gradient3d", "batch", "job3d"])
    por = round(rng.uniform(0.3, 0.7), 3)
    if kind in ("flow2d", "solute2d"):
        LX, LY = _between(rng, 32, 1100), _between(rng, 32, 1100)
        cap = (2e8 if kind == "flow2d" else 5e7) / (LX * LY)
        steps = 2 * _between(rng, 10, max(11, min(500, cap / 2)))
        return dict(kind=kind, LX=LX, LY=LY, real=rng.choice([8, 8, 8, 4]),
                    porosity=max(por, 0.5), radius=rng.randint(3, 9), steps=steps)
    if kind == "batch":
        low = _between(rng, 24, 64)
        return dict(kind=kind, samples=rng.randint(6, 24), low=low, high=rng.randint(low + 1, 96),
                    real=rng.choice([4, 4, 8]), steps=2 * _between(rng, 10, 60))
    lo, hi, budget = dict(flow3d=(24, 360, 1.5e9), open3d=(24, 256, 2e8), through3d=(24, 240, 6e8),
                          gradient3d=(24, 120, 1e8), job3d=(24, 200, 3e8))[kind]
    LX, LY, LZ = (_between(rng, lo, hi) for _ in range(3))
    cap = budget / (LX * LY * LZ)
    case = dict(kind=kind, LX=LX, LY=LY, LZ=LZ, real=rng.choice([4, 4, 8]),
                steps=2 * _between(rng, 8, max(9, min(60, cap / 2))))
    if kind != "open3d":
        case.update(porosity=por, radius=rng.randint(3, 8))
    if kind in ("flow3d", "open3d", "job3d"):
        case["model"] = rng.choice(["shifted", "shifted", "plain"]) if case["real"] == 8 else "shifted"
    if kind == "gradient3d":
        case["every"] = rng.choice([8, 16, 25])
    return case


# ---- inputs ----------------------------------------------------------------------

def _pack(ext, radius, porosity, rng):
    """Overlapping balls (discs in 2D) at random centres, as many as leave
    `porosity` on average; periodic.  ext = (LX, LY, LZ)."""
    LX, LY, LZ = ext
    r = np.arange(-radius, radius + 1)
    dz, dy, dx = np.meshgrid(r if LZ > 1 else np.zeros(1, int), r, r, indexing="ij")
    ball = dx * dx + dy * dy + dz * dz <= radius * radius
    ball = [torch.from_numpy(np.ascontiguousarray(v[ball])).cuda() for v in (dx, dy, dz)]
    n = max(1, math.ceil(math.log(1 / porosity) * LX * LY * LZ / ball[0].numel()))
    at = torch.from_numpy(np.stack([rng.integers(0, e, n) for e in ext])).cuda()
    solid = torch.zeros(LX * LY * LZ, dtype=torch.uint8, device="cuda")
    for c in torch.split(at, max(1, 20_000_000 // ball[0].numel()), dim=1):
        x, y, z = ((c[q][:, None] + ball[q][None]) % ext[q] for q in range(3))
        solid[(x + LX * (y + LY * z)).reshape(-1)] = 1
    return solid


def _mask(case, rng):
    ext = (case["LX"], case["LY"], case.get("LZ", 1))
    if case["kind"] == "open3d":
        # a channel: one wall plane, and a sill of random height on it
        solid = torch.zeros((ext[2], ext[1], ext[0]), dtype=torch.uint8, device="cuda")
        solid[:, 0] = 1
        at = int(rng.integers(0, max(1, ext[0] - 4)))
        solid[:, 1:1 + int(rng.integers(1, max(2, ext[1] // 4))), at:at + 2] = 1
        return solid.reshape(-1)
    solid = _pack(ext, case["radius"], case["porosity"], rng)
    if case["kind"] in ("flow2d", "solute2d"):       # reservoir rows at the faces
        solid.view(ext[1], ext[0])[0] = 0
        solid.view(ext[1], ext[0])[-1] = 0
    if case["kind"] in ("through3d", "gradient3d"):   # reservoir planes at the faces
        solid.view(ext[2], -1)[0] = 0
        solid.view(ext[2], -1)[-1] = 0
    return solid


def _params(case):
    """The run's parameters: those of the repository's configurations."""
    kind = case["kind"]
    two = kind in ("flow2d", "solute2d")
    p = dict(dims=2 if two else 3, LX=case["LX"], LY=case["LY"], LZ=case.get("LZ", 1),
             precision=case["real"], tau=(0.8, 1.0))
    if two:
        p.update(tau=(1.0, 0.8), pressure_s_in=(1, 0), pressure_n_out=(1, 0), rho_in=1.001,
                 rho_out=1.0)
    if kind in ("flow3d", "open3d", "job3d"):
        p.update(gaccel=(1e-6, 0, 0, 0, 0, 0))
        if case["model"] == "plain":
            p.update(accurate=0, compressible=1)
    if kind == "solute2d":
        p.update(nsubs=2, sigma_t_on=0, sigma_t_off=1 << 30, zeroconcgrad_n=1, sink=1e-4)
    if kind == "through3d":
        p.update(nsubs=2, tau=(0.9, 0.7), sigma_t_on=0, sigma_t_off=1 << 30,
                 pressure_b_in=(1, 0), pressure_t_out=(1, 0), rho_in=1.0005, rho_out=1.0,
                 constcon_b_in=1, zeroconcgrad_t=1, rho_sigma_in=1.0)
    if kind == "gradient3d":
        p.update(nsubs=2, tau=(0.8, 0.75), gaccel=(1e-5, 0, 0, 0, 0, 0), sigma_t_on=0,
                 sigma_t_off=1 << 30, constcon_b_in=1, zeroconcgrad_t=1, rho_sigma_in=1.0)
    return lbx.Params(**p)


def _plume(case, rng):
    """An initial concentration: a box of C = 1 over a background, smooth noise in it."""
    ext = [case.get("LZ", 1), case["LY"], case["LX"]]
    c = np.full(ext, 0.05)
    c[tuple(slice(e // 4, e // 4 + max(1, e // 2)) for e in ext)] = 1.0
    return (c * rng.uniform(0.9, 1.1, (ext[0], ext[1], 1))).reshape(-1)


def _objective(case):
    """The plane objective of the fit: a plane near the inlet over the last half of the run."""
    return dict(plane=min(6, case["LZ"] // 3), t_first=case["steps"] // 2 + 1,
                t_last=case["steps"], w_c=1.0, w_ux=10.0)


def _samples(case, seed):
    """(params, mask, tau) of each sample of a batch."""
    rng = np.random.default_rng(seed)
    edges = np.random.default_rng([case["low"], case["high"]])   # the study's images: fixed sizes
    for _ in range(case["samples"]):
        n = int(edges.integers(case["low"], case["high"] + 1))
        tau = float(rng.uniform(0.6, 1.2))
        por, radius = float(rng.uniform(0.3, 0.7)), int(rng.integers(3, 7))
        yield (lbx.Params(dims=3, LX=n, LY=n, LZ=n, precision=case["real"], tau=(tau, 1.0),
                          gaccel=(1e-6, 0, 0, 0, 0, 0)),
               _pack((n, n, n), radius, por, rng))


_STREAM = []


def _stream():
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


class _Fields:
    """A domain's macroscopic fields as torch sees them; a tensor made of this
    keeps it, and with it the domain that owns the memory."""

    def __init__(self, dom, shape, dtype):
        self.dom = dom
        ptr = dom.device_mv_ptr()
        self.__cuda_array_interface__ = dict(shape=shape, typestr=np.dtype(dtype).str,
                                             data=(ptr, False), version=3, strides=None)


def prepare(case, seed):
    if case["kind"] == "batch":
        made = list(_samples(case, seed))
        b = Batch([p for p, _ in made], [m.cpu().numpy() for _, m in made])
        b.set_stream(_stream())
        for i in range(len(made)):
            b.init_equilibrium(i, 1.0)
        return dict(case=case, batch=b, t=0)
    rng = np.random.default_rng(seed)
    p = _params(case)
    mask = _mask(case, rng).cpu().numpy()
    d = lbx.Domain(p, mask)
    d.set_stream(_stream())
    state = dict(case=case, dom=d, t=0, p=p)
    state["rho"] = np.ones(p.NN, p.dtype)
    if p.nsubs == 2:
        state["C"] = (np.zeros(p.NN) if case["kind"] == "through3d" else _plume(case, rng)).astype(p.dtype)
    if case["kind"] == "gradient3d":
        d.set_face_profile(False, rng.uniform(0.0, 1.0, p.LX * p.LY))
    if case["kind"] == "through3d":
        d.btc_start(p.LZ - 1, 1 << 16)
    d.init_equilibrium(0, state["rho"])
    if p.nsubs == 2:
        d.init_equilibrium(1, state["C"])
    mv = torch.as_tensor(_Fields(d, (p.nsubs, 1 + p.dims, p.NN), p.dtype), device="cuda")
    state["fields"] = dict(rho=mv[0, 0], u=mv[0, 1:])
    if p.nsubs == 2:
        state["fields"]["C"] = mv[1, 0]
    return state


# ---- one pass --------------------------------------------------------------------

def run(state):
    case, steps = state["case"], state["case"]["steps"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.run(state["t"], steps, steps)
        state["t"] += steps
        mv = [b.download_mv(i) for i in range(case["samples"])]
        return dict(rho=np.concatenate([m[0] for m in mv]),
                    u=np.concatenate([m[1:] for m in mv], axis=1))
    d = state["dom"]
    if case["kind"] == "gradient3d":
        d.init_equilibrium(0, state["rho"])
        d.init_equilibrium(1, state["C"])
        J = d.adjoint_forward(0, steps, case["every"], **_objective(case))
        g = d.adjoint_backward(profile_b=True)
        return dict(J=J, d_gaccel=np.array(g["d_gaccel"]), d_tau=g["d_tau"],
                    d_tau_s=g["d_tau_s"], d_profile=g["d_profile_b"])
    if case["kind"] == "job3d":
        d.init_equilibrium(0, state["rho"])
        d.run(0, steps, steps)
        mv = d.download_mv()
        return dict(rho=mv[0, 0], u=mv[0, 1:])
    d.run(state["t"], steps, steps)
    state["t"] += steps
    return state["fields"]


def work(case):
    """A time step reads and writes every population of every fluid node; a
    reverse step of the adjoint reads the forward state and reads and writes
    the adjoint one, and needs the forward step again."""
    if case["kind"] == "batch":
        edges = np.random.default_rng([case["low"], case["high"]])
        nodes = 0.5 * sum(int(edges.integers(case["low"], case["high"] + 1)) ** 3
                          for _ in range(case["samples"]))
        return dict(bytes=nodes * 38 * case["real"] * case["steps"], flops=nodes * 230 * case["steps"])
    q = 9 if case["kind"] in ("flow2d", "solute2d") else 19
    subs = 2 if case["kind"] in ("solute2d", "through3d", "gradient3d") else 1
    nodes = case["LX"] * case["LY"] * case.get("LZ", 1) * case.get("porosity", 0.97)
    sweeps = (1 + 1 + 1.5) if case["kind"] == "gradient3d" else 1
    return dict(bytes=sweeps * nodes * subs * 2 * q * case["real"] * case["steps"],
                flops=sweeps * nodes * subs * 12 * q * case["steps"])


# ---- the same in 64 bits ---------------------------------------------------------

class _Plain:
    """The lattice over its fluid nodes: `d = pull(f)` streams with half-way
    bounce-back (from the populations after a collision), the faces rewrite
    the unknowns, `flow` and `solute` collide."""

    def __init__(self, p, solid):
        self.p = p
        self.Q = p.Q
        LX, LY, LZ = p.LX, p.LY, p.LZ
        solid = solid.bool()
        node = torch.nonzero(~solid).reshape(-1)
        self.node, self.F = node, node.numel()
        rank = torch.cumsum((~solid).to(torch.int64), 0) - 1
        x, y, z = node % LX, (node // LX) % LY, node // (LX * LY)
        own = torch.arange(self.F, device="cuda")
        src = []
        for a in range(self.Q):
            cx, cy, cz = _C[a]
            up = (x - cx) % LX + LX * ((y - cy) % LY + LY * ((z - cz) % LZ))
            src.append(torch.where(solid[up], _opp(a) * self.F + own, a * self.F + rank[up])
                       .to(torch.int32 if self.Q * self.F < 2 ** 31 else torch.int64))
        self.src = torch.cat(src)
        self.w = _W2 if self.Q == 9 else _W3
        line = y if p.dims == 2 else z
        self.low = int((line == 0).sum())
        self.high = int((line == (LY if p.dims == 2 else LZ) - 1).sum())

    def pull(self, f):
        return f.reshape(-1).index_select(0, self.src).view(self.Q, self.F)

    def at_faces(self, d, low, high):
        """d with the face rules applied to its first and last plane (row)."""
        parts = [d]
        if low or high:
            a, b = self.low, self.F - self.high
            parts = [d[:, :a], d[:, a:b], d[:, b:]]
            for part, rules in ((0, low), (2, high)):
                for rule in rules:
                    parts[part] = torch.stack(rule(list(parts[part])))
        return torch.cat(parts, dim=1)

    def axis(self, a):
        return _C[a][1] if self.p.dims == 2 else _C[a][2]

    def unknown(self, high):
        return [a for a in range(self.Q) if self.axis(a) == (-1 if high else 1)]

    def pressure(self, high, drho):
        def rule(d):
            d = list(d)
            flat = sum(d[a] for a in range(self.Q) if self.axis(a) == 0)
            out = sum(d[a] for a in range(self.Q) if self.axis(a) == (1 if high else -1))
            # the momentum into the lattice across the face
            J = drho - (flat + 2 * out)
            n = [0.5 * (sum(d[a] * _C[a][q] for a in range(self.Q) if self.axis(a) == 0))
                 for q in range(2)]
            new = {}
            for a in self.unknown(high):
                cx, cy = _C[a][0], (0 if self.p.dims == 2 else _C[a][1])
                if cx == 0 and cy == 0:
                    new[a] = d[_opp(a)] + J * (2 / 3 if self.p.dims == 2 else 1 / 3)
                else:
                    new[a] = d[_opp(a)] + J / 6 - (cx * n[0] + cy * n[1])
            for a, v in new.items():
                d[a] = v
            return d
        return rule

    def concentration(self, high, conc):
        def rule(d):
            un = self.unknown(high)
            X = (conc - sum(d[a] for a in range(self.Q) if a not in un)) / sum(self.w[a] for a in un)
            return [self.w[a] * X if a in un else d[a] for a in range(self.Q)]
        return rule

    def zero_gradient(self, high):
        def rule(d):
            un = self.unknown(high)
            X = sum(d[_opp(a)] for a in un) / sum(self.w[a] for a in un)
            return [self.w[a] * X if a in un else d[a] for a in range(self.Q)]
        return rule

    def cu(self, a, u):
        s = None
        for q in range(self.p.dims):
            if _C[a][q]:
                v = u[q] if _C[a][q] > 0 else -u[q]
                s = v if s is None else s + v
        return s

    def flow(self, d, tau, g):
        """(rho as reported, u, populations after the collision)"""
        rho = d.sum(0)
        rA = 1.0 if self.p.accurate else 0.0
        den = rho if not self.p.accurate else 1.0
        u = []
        for q in range(self.p.dims):
            m = sum(d[a] if _C[a][q] > 0 else -d[a] for a in range(self.Q) if _C[a][q])
            u.append(m / den + tau * g[q])
        usq = sum(v * v for v in u)
        out = []
        for a in range(self.Q):
            c = self.cu(a, u)
            poly = -1.5 * usq if c is None else 3 * c + 4.5 * c * c - 1.5 * usq
            out.append(d[a] + (self.w[a] * (rho + den * poly) - d[a]) / tau)
        return rho + rA, u, torch.stack(out)

    def solute(self, d, u, tau, scale):
        C = d.sum(0) * scale
        out = []
        for a in range(self.Q):
            c = self.cu(a, u)
            out.append(d[a] + (self.w[a] * C * (1 if c is None else 1 + 3 * c) - d[a]) / tau)
        return C, torch.stack(out)


def _faces(case, L, profile=None):
    """(flow low, flow high, solute low, solute high) face rules."""
    p, kind = L.p, case["kind"]
    if kind in ("flow2d", "solute2d", "through3d"):
        lo, hi = [L.pressure(False, p.rho_in - 1.0)], [L.pressure(True, p.rho_out - 1.0)]
    else:
        lo = hi = []
    if kind == "solute2d":
        return lo, hi, [], [L.zero_gradient(True)]
    if kind in ("through3d", "gradient3d"):
        c = p.rho_sigma_in if profile is None else profile
        return lo, hi, [L.concentration(False, c)], [L.zero_gradient(True)]
    return lo, hi, [], []


def _start(L, C0=None):
    """Populations at rest at rho = 1 (deviations, or whole), and the solute's."""
    w = torch.tensor(L.w, dtype=torch.float64, device="cuda")[:, None]
    f = torch.zeros((L.Q, L.F), dtype=torch.float64, device="cuda")
    if not L.p.accurate:
        f = f + w
    return f, None if C0 is None else w * C0[L.node]


def _fields(case, p, solid, C0=None, rho0=1.0):
    """rho, u and C after one pass from the start, over all nodes (solid ones keep the start's)."""
    L = _Plain(p, solid)
    f, g = _start(L, C0)
    flo, fhi, slo, shi = _faces(case, L)
    s1 = 1.0 - p.sink * p.tau[1]
    rho = u = C = None
    for t in range(1, case["steps"] + 1):
        rho, u, f = L.flow(L.at_faces(L.pull(f), flo, fhi), p.tau[0], p.gaccel[:3])
        if g is not None:
            C, g = L.solute(L.at_faces(L.pull(g), slo, shi), u, p.tau[1], s1 if t % 2 else s1 * s1)

    def whole(v, base):
        out = base.clone()
        out[L.node] = v
        return out

    zero = torch.zeros(p.NN, dtype=torch.float64, device="cuda")
    out = dict(rho=whole(rho, zero + rho0), u=torch.stack([whole(v, zero) for v in u]))
    if g is not None:
        out["C"] = whole(C, C0)
    return out


def _gradient(case, p, solid, C0, profile):
    L = _Plain(p, solid)
    f, g = _start(L, C0)
    gacc = torch.tensor(p.gaccel[:3], dtype=torch.float64, device="cuda", requires_grad=True)
    tau = [torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in p.tau]
    prof = profile.clone().requires_grad_(True)
    o = _objective(case)
    z = L.node // (p.LX * p.LY)
    plane = torch.nonzero(z == o["plane"]).reshape(-1)
    n = o["t_last"] - o["t_first"] + 1

    def stretch(f, g, t0, t1):
        J = torch.zeros((), dtype=torch.float64, device="cuda")
        flo, fhi, slo, shi = _faces(case, L, prof)
        for t in range(t0, t1):
            _, u, f = L.flow(L.at_faces(L.pull(f), flo, fhi), tau[0], gacc)
            C, g = L.solute(L.at_faces(L.pull(g), slo, shi), u, tau[1], 1.0)
            if o["t_first"] <= t <= o["t_last"]:
                J = J + (o["w_c"] * C[plane].mean() + o["w_ux"] * u[0][plane].mean()) / n
        return f, g, J

    # reverse sweep over stored states
    every = 5
    ts = list(range(1, case["steps"] + 1, every))
    kept, J = [], 0.0
    for t in ts:
        kept.append((f, g))
        with torch.no_grad():
            f, g, j = stretch(f, g, t, min(t + every, case["steps"] + 1))
        J += float(j)
    lf, lg = torch.zeros_like(f), torch.zeros_like(g)
    total = [torch.zeros_like(v) for v in (gacc, tau[0], tau[1], prof)]
    for t, (f, g) in zip(reversed(ts), reversed(kept)):
        f, g = f.detach().requires_grad_(True), g.detach().requires_grad_(True)
        f1, g1, j = stretch(f, g, t, min(t + every, case["steps"] + 1))
        parts = torch.autograd.grad((f1 * lf).sum() + (g1 * lg).sum() + j,
                                    (f, g, gacc, tau[0], tau[1], prof), allow_unused=True)
        lf, lg = parts[0], parts[1]
        for v, d in zip(total, parts[2:]):
            if d is not None:
                v += d
    return dict(J=J, d_gaccel=total[0], d_tau=float(total[1]), d_tau_s=float(total[2]),
                d_profile=total[3])


def exact(case, seed):
    if case["kind"] == "batch":
        # a batch's macroscopic fields hold 0 on solid nodes
        got = [_fields(case, p, m, rho0=0.0) for p, m in _samples(case, seed)]
        return dict(rho=torch.cat([v["rho"] for v in got]), u=torch.cat([v["u"] for v in got], dim=1))
    rng = np.random.default_rng(seed)
    p = _params(case)
    solid = _mask(case, rng)
    C0 = None
    if p.nsubs == 2:
        C0 = np.zeros(p.NN) if case["kind"] == "through3d" else _plume(case, rng)
        C0 = torch.from_numpy(C0.astype(p.dtype).astype(np.float64)).cuda()
    if case["kind"] == "gradient3d":
        prof = rng.uniform(0.0, 1.0, p.LX * p.LY).astype(p.dtype).astype(np.float64)
        return _gradient(case, p, solid, C0, torch.from_numpy(prof).cuda())
    return _fields(case, p, solid, C0)
