"""The work that a user of this library has it do, as cases that can be timed.

Each case is one pass through the public Python entry points (``Box``,
``System``, ``Batch``, ``surrogate.Mlp``): the reference's drivers keep a
simulation in host arrays between chunks of steps (snapshots, frames written
to disk), so a pass takes host arrays in and gives host arrays back wherever
such a driver does.  The kinds:

  frame     a driver's loop body: a few steps, then the frame and the order
            parameter (Box.Multi_Step + Box.Save).  The smallest call.
  series    discrete Vicsek, the polarization after every `every` steps.
  vicsek    a chunk of discrete Vicsek steps (dt = 1).
  abp       a chunk of repulsive active Brownian steps (Verlet list).
  vesicles  a chunk of ring vesicles with swimmers (bonds, bending, R12).
  lyapunov  base and tangent dynamics with renormalisations.
  sweep     a batch of independent Vicsek systems, uploaded and read back.
  sweepon   a running batch: steps and a poll of every point's statistics.
  fit       the sweep's surrogate: training of the ensemble, then predictions.
  pairs     pair statistics of a frame: g(r) and the body-frame histogram.

``exact`` restates the noise (Philox4x32-10, Salmon et al., SC'11) and the
equations in 64 bits with torch, from the model definitions alone.
"""
import ctypes
import math

import numpy as np
import torch

from spp_gb300 import Batch, System, abi, configs, surrogate
from spp_gb300.system import Box

DEV = "cuda"


def listed():
    return [
        # a reference-shaped driver that writes a frame after every step (a
        # movie of a small box): launches and host round trips are all there is
        {"name": "frame_1000", "kind": "frame", "n": 1000, "rho": 1.0, "integrator": "rk2", "every": 1},
        # the plain Vicsek workload of configs.vicsek_config: P after every step
        {"name": "series_4096", "kind": "series", "n": 4096, "rho": 1.0, "model": "vector_sum", "eta": 0.3,
         "frames": 100, "every": 1},
        # the reference's own angle average, a system past one cluster's reach
        {"name": "vicsek_50001", "kind": "vicsek", "n": 50001, "rho": 1.0, "model": "ref_angle", "eta": 0.2,
         "steps": 10},
        # the largest system that the library gathers with four lanes
        {"name": "abp_16384", "kind": "abp", "n": 16384, "rho": 1.0, "integrator": "rk2", "law": "harmonic",
         "steps": 100},
        # a mid-sized odd system with the reference's force law and RK4
        {"name": "abp_65537_r12", "kind": "abp", "n": 65537, "rho": 0.8, "integrator": "rk4", "law": "r12",
         "steps": 50},
        # the headline workload (configs.abp_config, bench.py): one 200-step chunk
        {"name": "abp_1m", "kind": "abp", "n": 1 << 20, "rho": 1.0, "integrator": "rk2", "law": "harmonic",
         "steps": 200},
        # configs.vesicle_config: 1024 rings of 128 beads, 32 swimmers each
        {"name": "vesicles_164k", "kind": "vesicles", "rings": 1024, "ring_size": 128, "swimmers": 32,
         "integrator": "rk4", "steps": 50},
        # configs.lyapunov_config with a flocked start (its long-run state)
        {"name": "lyapunov_16384", "kind": "lyapunov", "n": 16384, "rho": 1.0, "k": 8, "steps": 50,
         "every": 10, "clump": 0.6},
        # a part of configs.sweep_points: state in, a window of steps, state out
        {"name": "sweep_64", "kind": "sweep", "points": 64, "n_max": 65536, "steps": 100},
        # the whole 512-point sweep while it runs: steps and the statistics
        {"name": "sweep_512_running", "kind": "sweepon", "points": 512, "n_max": 65536, "steps": 32},
        # a fit of the sweep's surrogate on the completed points, and its answers
        {"name": "fit_300", "kind": "fit", "ensemble": 5, "samples": 300, "iters": 300, "queries": 512},
        # pair statistics of a saved frame
        {"name": "pairs_262144", "kind": "pairs", "n": 262144, "rho": 1.0, "r_max": 5.0, "nbins": 50,
         "lx": 3.0, "ly": 3.0, "gx": 60, "gy": 60},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["frame", "series", "vicsek", "abp", "abp", "abp", "vesicles", "lyapunov", "sweep", "fit",
                       "pairs"])
    rho = round(rng.uniform(0.25, 1.2), 3)
    if kind == "frame":
        return {"kind": kind, "n": _log(rng, 300, 20000), "rho": rho, "integrator": rng.choice(["rk2", "rk4"]),
                "every": rng.choice([1, 2, 5])}
    if kind == "series":
        return {"kind": kind, "n": _log(rng, 1000, 60000), "rho": round(rng.uniform(0.25, 2.0), 3),
                "model": "vector_sum", "eta": round(rng.uniform(0.05, 0.6), 3), "frames": rng.randint(20, 100),
                "every": rng.choice([1, 1, 5])}
    if kind == "vicsek":
        return {"kind": kind, "n": _log(rng, 2000, 500000), "rho": round(rng.uniform(0.25, 2.0), 3),
                "model": rng.choice(["vector_sum", "ref_angle", "ref_vector"]),
                "eta": round(rng.uniform(0.05, 0.6), 3), "steps": rng.randint(5, 10)}
    if kind == "abp":
        law = rng.choice(["harmonic", "harmonic", "r12"])
        return {"kind": kind, "n": _log(rng, 1000, 1 << 20), "rho": min(rho, 0.8) if law == "r12" else rho,
                "integrator": rng.choice(["euler", "rk2", "rk2", "rk4"]), "law": law, "steps": rng.randint(20, 100)}
    if kind == "vesicles":
        size = rng.choice([48, 64, 100, 128])
        return {"kind": kind, "rings": _log(rng, 20, 131072 // size), "ring_size": size,
                "swimmers": rng.randint(0, size // 8), "integrator": rng.choice(["rk2", "rk4"]),
                "steps": rng.randint(20, 60)}
    if kind == "lyapunov":
        return {"kind": kind, "n": _log(rng, 1000, 24000), "rho": round(rng.uniform(0.5, 1.2), 3),
                "k": rng.randint(1, 8), "steps": rng.randint(10, 40), "every": rng.choice([5, 10]),
                "clump": round(rng.uniform(0.0, 0.6), 3)}
    if kind == "sweep":
        return {"kind": kind, "points": _log(rng, 8, 100), "n_max": _log(rng, 8192, 65536),
                "steps": rng.randint(20, 100)}
    if kind == "fit":
        return {"kind": kind, "ensemble": rng.randint(3, 8), "samples": rng.randint(60, 500),
                "iters": rng.randint(50, 300), "queries": rng.randint(64, 512)}
    return {"kind": kind, "n": _log(rng, 4096, 1 << 20), "rho": rho, "r_max": round(rng.uniform(2.0, 6.0), 2),
            "nbins": rng.randint(20, 200), "lx": round(rng.uniform(1.5, 4.0), 2),
            "ly": round(rng.uniform(1.5, 4.0), 2), "gx": rng.randint(10, 80), "gy": rng.randint(10, 80)}


# ------------------------------------------------------------------ inputs
INTEGRATORS = {"euler": abi.INT_EULER, "rk2": abi.INT_RK2, "rk4": abi.INT_RK4}
VICSEK = {"vector_sum": abi.MODEL_VICSEK, "ref_angle": abi.MODEL_VICSEK_REF_ANGLE,
          "ref_vector": abi.MODEL_VICSEK_REF_VECTOR}


def _box(n, rho):
    return 0.5 * math.sqrt(n / rho)


def _f32_in_box(v, L):
    v = v.astype(np.float32)
    return np.where(v >= np.float32(L), -np.float32(L), v).astype(np.float32)


def _uniform(n, L, g):
    """Uniform positions and headings, the configured start of a run."""
    x = _f32_in_box((2.0 * g.random(n) - 1.0) * L, L)
    y = _f32_in_box((2.0 * g.random(n) - 1.0) * L, L)
    return x, y, ((2.0 * g.random(n) - 1.0) * math.pi).astype(np.float32)


def _lattice(n, L, g):
    """A square lattice with a little jitter: no two disks overlap hard, as
    the r^-12 law needs (the reference starts such runs from a lattice)."""
    m = int(math.ceil(math.sqrt(n)))
    a = 2.0 * L / m
    site = g.permutation(m * m)[:n]
    x = -L + (site % m + 0.5 + 0.08 * (2.0 * g.random(n) - 1.0)) * a
    y = -L + (site // m + 0.5 + 0.08 * (2.0 * g.random(n) - 1.0)) * a
    return _f32_in_box(x, L), _f32_in_box(y, L), ((2.0 * g.random(n) - 1.0) * math.pi).astype(np.float32)


def _flocked(n, L, clump, g):
    """A flocked state: a fraction `clump` of the particles in round flocks of
    a few hundred with a common heading, the rest uniform."""
    x, y, th = _uniform(n, L, g)
    m = int(clump * n)
    if m:
        nf = max(1, m // 400)
        which = g.integers(0, nf, m)
        cx, cy, ct = (2 * g.random((3, nf)) - 1.0) * np.array([[L], [L], [math.pi]])
        r = 3.5 * np.sqrt(g.random(m))
        a = 2 * math.pi * g.random(m)
        fx = cx[which] + r * np.cos(a)
        fy = cy[which] + r * np.sin(a)
        ft = ct[which] + 0.3 * g.standard_normal(m)
        x[:m] = _f32_in_box(fx - 2 * L * np.floor((fx + L) / (2 * L)), L)
        y[:m] = _f32_in_box(fy - 2 * L * np.floor((fy + L) / (2 * L)), L)
        th[:m] = (ft - 2 * math.pi * np.floor(ft / (2 * math.pi) + 0.5)).astype(np.float32)
    return x, y, th


def _abp_params(case, seed):
    n = case["n"]
    if case.get("law") == "r12":
        p = configs.reference_defaults(abi.MODEL_ABP)   # RepulsiveParticle's own statics
        p.n, p.L, p.seed = n, _box(n, case["rho"]), seed
        p.Dr, p.dt, p.skin = 0.1, 0.002, 0.3
        p.integrator = INTEGRATORS[case["integrator"]]
        return p
    return configs.abp_config(n=n, L=_box(n, case["rho"]), seed=seed, integrator=INTEGRATORS[case["integrator"]])


def _params(case, seed):
    kind = case["kind"]
    if kind in ("frame", "abp"):
        return _abp_params(case, seed)
    if kind in ("series", "vicsek"):
        return configs.vicsek_config(n=case["n"], L=_box(case["n"], case["rho"]), eta=case["eta"], seed=seed,
                                     model=VICSEK[case["model"]])
    if kind == "vesicles":
        return configs.vesicle_config(n_rings=case["rings"], ring_size=case["ring_size"],
                                      swimmers_per_ring=case["swimmers"], seed=seed,
                                      integrator=INTEGRATORS[case["integrator"]])
    if kind == "lyapunov":
        return configs.lyapunov_config(n=case["n"], rho=case["rho"], seed=seed)
    return configs.abp_config(n=case["n"], L=_box(case["n"], case["rho"]), seed=seed)   # pairs


def _state(case, p, seed):
    g = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "vesicles":
        return configs.vesicle_state(p, seed=seed)
    if kind == "abp" and case["law"] == "r12":
        return _lattice(p.n, p.L, g)
    if kind == "lyapunov":
        return _flocked(p.n, p.L, case["clump"], g)
    if kind == "pairs":
        return _flocked(p.n, p.L, 0.3, g)
    return _uniform(p.n, p.L, g)


def _fit_data(case, seed):
    """Standardised features (parameters and moments of P over the window) and
    targets in [0, 1] of completed sweep points, K-fold bagging weights."""
    g = np.random.default_rng(seed)
    B, E = case["samples"], case["ensemble"]
    x = g.standard_normal((B + case["queries"], 7)).astype(np.float32)
    t = (0.5 + 0.5 * np.tanh(0.7 * x[:B, 0] - x[:B, 1] + 0.3 * x[:B, 2] * x[:B, 3])
         + 0.02 * g.standard_normal(B)).astype(np.float32)
    w = (np.arange(B)[None, :] % E != np.arange(E)[:, None]).astype(np.float32)
    u = 2.0 * g.random((E, surrogate.n_params())) - 1.0
    H = surrogate.HIDDEN
    theta = np.zeros((E, surrogate.n_params()), np.float32)
    o = H * 7
    theta[:, :o] = u[:, :o] / math.sqrt(7)
    theta[:, o + H:o + H + H * H] = u[:, o + H:o + H + H * H] / math.sqrt(H)
    o += H + H * H + H
    theta[:, o:o + H] = u[:, o:o + H] / math.sqrt(H)
    return {"x": x[:B], "t": t, "w": w, "theta": theta, "xq": x[B:]}


def _sweep(case, seed):
    pts = configs.sweep_points(n_points=case["points"], n_max=case["n_max"])   # the sweep's own points
    g = np.random.default_rng(seed)
    for q in pts:
        q.seed = seed
    parts = [_uniform(p.n, p.L, g) for p in pts]
    return pts, tuple(np.concatenate([q[c] for q in parts]) for c in range(3))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind == "fit":
        s.data = _fit_data(case, seed)
        s.mlp = surrogate.Mlp(ensemble=case["ensemble"], seed=seed)
        return s
    if kind in ("sweep", "sweepon"):
        pts, s.start = _sweep(case, seed)
        s.batch = Batch(pts)
        s.batch.set_windows(50, 50, 0)
        if kind == "sweepon":
            s.batch.upload(*s.start)
        return s
    p = _params(case, seed)
    s.start = _state(case, p, seed)
    if kind == "frame":
        s.box = Box(p)
        s.box.Init(*s.start)
        return s
    s.system = System(p)
    if kind == "pairs":
        s.system.upload(*s.start)
    s.seed = seed
    return s


# ------------------------------------------------------------------ one pass
STATS = [f for f, _ in abi.SppSweepStats._fields_ if f != "reserved"]


def _stats(polled):
    a = np.ctypeslib.as_array((abi.SppSweepStats * len(polled))(*polled)) if polled else None
    return {f: np.ascontiguousarray(a[f]) for f in STATS}


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "frame":
        s.box.Multi_Step(case["every"])
        snap = s.box.Save()
        return {"x": snap.x, "y": snap.y, "theta": snap.theta, "img_x": snap.img_x, "img_y": snap.img_y,
                "P": s.box.Compute_Polarization(), "step": snap.step}
    if kind == "fit":
        d = s.data
        s.mlp.set_params(d["theta"])
        loss = s.mlp.train(d["x"], d["t"], iters=case["iters"], lr=1e-3, weights=d["w"])
        return {"loss": loss, "params": s.mlp.params(), "y": s.mlp.predict(d["xq"])}
    if kind == "sweep":
        s.batch.upload(*s.start)
        s.batch.step(case["steps"])
        out = _stats(s.batch.poll())
        out["state"] = s.batch.download()
        return out
    if kind == "sweepon":
        s.batch.step(case["steps"])
        return _stats(s.batch.poll())
    if kind == "pairs":
        return {"g": s.system.radial_distribution(case["r_max"], case["nbins"]).astype(np.int64),
                "body": s.system.pair_distribution(case["lx"], case["ly"], case["gx"],
                                                   case["gy"]).astype(np.int64)}
    s.system.upload(*s.start)
    if kind == "series":
        p, px, py = s.system.polarization_series(case["frames"], case["every"])
        return {"p": p, "px": px, "py": py, "state": s.system.download()}
    if kind == "lyapunov":
        s.system.lyap_init(case["k"], seed=s.seed)
        s.system.lyap_step(case["steps"], case["every"])
        lam, span = s.system.lyap_exponents()
        return {"lambda": lam, "span": span, "vectors": s.system.lyap_vectors(), "state": s.system.download()}
    s.system.step(case["steps"])
    return {"state": s.system.download()}


# ------------------------------------------------------------------ work
STAGES = {"euler": 1, "rk2": 2, "rk4": 4}


def work(case):
    """Bytes: host inputs once and outputs once, and for each step the state
    read once and written once (x, y, theta: 12 bytes each way; a step needs
    the whole of the one before).  Operations: per stage about 100 for a
    particle's own update and noise, 25 for each ordered pair in range."""
    kind = case["kind"]
    if kind == "fit":
        P = surrogate.n_params()
        fb = 6.0 * P * case["samples"]
        return {"bytes": 4.0 * (case["ensemble"] * (2 * P + case["samples"] + case["queries"])
                                + 8 * case["samples"] + 7 * case["queries"]),
                "flops": case["ensemble"] * (case["iters"] * fb + 2.0 * P * (case["samples"] + case["queries"]))}
    if kind in ("sweep", "sweepon"):
        pts = configs.sweep_points(n_points=case["points"], n_max=case["n_max"])
        n = float(sum(p.n for p in pts))
        pairs = sum(p.n * p.n / (4.0 * p.L * p.L) * math.pi for p in pts)
        io = 32.0 * n if kind == "sweep" else 0.0
        return {"bytes": io + 24.0 * n * case["steps"] + ctypes.sizeof(abi.SppSweepStats) * len(pts),
                "flops": case["steps"] * (100.0 * n + 8.0 * pairs)}
    if kind == "pairs":
        n, rho = float(case["n"]), case["rho"]
        tested = n * rho * (math.pi * case["r_max"] ** 2 + 4 * case["lx"] * case["ly"])
        return {"bytes": 2 * 16.0 * n + 8.0 * (case["nbins"] + case["gx"] * case["gy"]), "flops": 15.0 * tested}
    if kind == "vesicles":
        n = float(case["rings"] * (case["ring_size"] + case["swimmers"]))
        steps, stages, near, per = case["steps"], STAGES[case["integrator"]], 2.0, 160.0
    else:
        n = float(case["n"])
        near, per = case["rho"] * math.pi, 100.0
        stages = STAGES.get(case.get("integrator"), 4 if kind == "lyapunov" else 1)
        steps = case["frames"] * case["every"] if kind == "series" else case.get("steps", case.get("every"))
    io = 32.0 * n + (20.0 * n if kind == "lyapunov" else 0.0)
    if kind == "frame":
        io = 20.0 * n
    tangent = case["k"] if kind == "lyapunov" else 0
    io += 12.0 * n * tangent
    return {"bytes": io + steps * n * 24.0 * (1 + tangent),
            "flops": steps * stages * n * (per * (1 + 0.3 * tangent) + near * (25.0 + 3.0 * tangent))}


# ------------------------------------------------------------------ 64 bits
def _philox(c, seed):
    """Philox4x32-10 on int64 tensors of 32-bit words; c: four counter words."""
    M = 0xFFFFFFFF
    c0, c1, c2, c3 = c
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57   # the product's 64 bits, as a signed word
        c0, c1, c2, c3 = ((p1 >> 32) & M) ^ c1 ^ k0, p1 & M, ((p0 >> 32) & M) ^ c3 ^ k1, p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _words(n, step, stream, seed):
    ids = torch.arange(n, dtype=torch.int64, device=DEV)
    z = torch.zeros_like(ids)
    return _philox((ids, z + step, z + stream, z), seed)


def _normal(n, step, stream, seed):
    a, b, _, _ = _words(n, step, stream, seed)
    u1 = ((a >> 8) + 1).double() * 2.0 ** -24
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos((b >> 8).double() * (2.0 ** -24 * 2 * math.pi))


def _wrap(v, L):
    return v - 2 * L * torch.floor((v + L) / (2 * L))


def _angle(t):
    return t - 2 * math.pi * torch.floor(t / (2 * math.pi) + 0.5)


def _near(x, y, L, r):
    """Ordered pairs (i, j), i != j, closer than r in the periodic box."""
    n = x.numel()
    D = max(1, int(2 * L / r))
    if D < 3:
        i = torch.arange(n, device=DEV).repeat_interleave(n)
        j = torch.arange(n, device=DEV).repeat(n)
        keep = i != j
        i, j = i[keep], j[keep]
    else:
        cx = ((x + L) * (D / (2 * L))).long().clamp(0, D - 1)
        cy = ((y + L) * (D / (2 * L))).long().clamp(0, D - 1)
        order = torch.argsort(cy * D + cx)
        count = torch.bincount(cy * D + cx, minlength=D * D)
        start = torch.cumsum(count, 0) - count
        got = []
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                c = ((cy + oy) % D) * D + (cx + ox) % D
                m = count[c]
                i = torch.arange(n, device=DEV).repeat_interleave(m)
                at = torch.arange(i.numel(), device=DEV) - (torch.cumsum(m, 0) - m).repeat_interleave(m)
                j = order[start[c][i] + at]
                dx, dy = _image(x[i] - x[j], L), _image(y[i] - y[j], L)
                keep = (dx * dx + dy * dy < r * r) & (i != j)
                got.append((i[keep], j[keep]))
        i, j = (torch.cat([g[q] for g in got]) for q in (0, 1))
    return i, j


def _image(d, L):
    return d - 2 * L * torch.floor((d + L) / (2 * L))


class _Near:
    """Pairs within r + skin, found again once a particle has moved skin / 4."""

    def __init__(self, L, r, skin=0.3):
        self.L, self.r, self.skin, self.at = L, r, skin, None

    def __call__(self, x, y):
        if self.at is not None:
            d = torch.maximum(_image(x - self.at[0], self.L).abs().max(), _image(y - self.at[1], self.L).abs().max())
            if float(d) < self.skin / 4:
                return self.at[2]
        self.at = (x.clone(), y.clone(), _near(x, y, self.L, self.r + self.skin))
        return self.at[2]


def _sum(n, i, v):
    return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, i, v)


def _rates_abp(p, near):
    """RepulsiveParticle / ContinuousParticle: velocity and turning rate."""
    def rates(x, y, th):
        n = x.numel()
        i, j = near(x, y)
        dx, dy = _image(x[i] - x[j], p.L), _image(y[i] - y[j], p.L)
        d = torch.sqrt(dx * dx + dy * dy)
        vx, vy = p.v0 * torch.cos(th), p.v0 * torch.sin(th)
        if p.force_law != abi.FORCE_NONE:
            if p.force_law == abi.FORCE_HARMONIC:
                f = p.k_rep * (1.0 - d / p.r_rep) / d
            else:
                f = p.k_rep * ((p.sigma_rep / d) ** 13 - (p.sigma_rep / p.r_rep) ** 13) / d
            f = torch.where((d < p.r_rep) & (d > 0), f, torch.zeros_like(f))
            vx, vy = vx + _sum(n, i, f * dx), vy + _sum(n, i, f * dy)
        if p.model == abi.MODEL_BEADS:
            return vx, vy, torch.zeros_like(th)
        al = d < p.r_align
        S = _sum(n, i[al], torch.sin(th[j[al]] - th[i[al]]))
        if p.model == abi.MODEL_CONTINUOUS:
            return vx, vy, p.g / math.pi * S
        if p.align_mode == abi.ALIGN_MEAN:
            return vx, vy, p.g * S / (1.0 + _sum(n, i[al], torch.ones_like(d[al])))
        return vx, vy, S * p.g / (math.pi * p.r_align ** 2)
    return rates


def _rates_vesicles(p, near):
    nb = p.n_rings * p.ring_size
    law = _rates_abp(p, near)

    def rates(x, y, th):
        pvx, pvy, _ = law(x, y, th)                       # v0 (cos, sin) + pair force
        fx, fy = pvx - p.v0 * torch.cos(th), pvy - p.v0 * torch.sin(th)
        bx, by = x[:nb].view(p.n_rings, -1), y[:nb].view(p.n_rings, -1)
        ux, uy = _image(bx - bx.roll(1, 1), p.L), _image(by - by.roll(1, 1), p.L)   # bond into bead m
        u = torch.sqrt(ux * ux + uy * uy)
        t = p.k_bond * (p.bond_rest / u - 1.0)
        gx, gy = t * ux - (t * ux).roll(-1, 1), t * uy - (t * uy).roll(-1, 1)
        wx, wy, w = ux.roll(-1, 1), uy.roll(-1, 1), u.roll(-1, 1)                   # bond out of bead m
        c = (ux * wx + uy * wy) / (u * w)
        dux, duy = wx / (u * w) - c * ux / u ** 2, wy / (u * w) - c * uy / u ** 2
        dwx, dwy = ux / (u * w) - c * wx / w ** 2, uy / (u * w) - c * wy / w ** 2
        gx = gx + p.kappa_bend * (dwx.roll(1, 1) + dux - dwx - dux.roll(-1, 1))
        gy = gy + p.kappa_bend * (dwy.roll(1, 1) + duy - dwy - duy.roll(-1, 1))
        fx, fy = fx.clone(), fy.clone()
        fx[:nb] += gx.reshape(-1)
        fy[:nb] += gy.reshape(-1)
        swim = torch.ones_like(th)
        swim[:nb] = 0.0
        return (p.v0 * swim * torch.cos(th) + p.mu * fx, p.v0 * swim * torch.sin(th) + p.mu * fy,
                torch.zeros_like(th))
    return rates


def _advance(p, rates, x, y, th, steps, still=0):
    """`steps` steps of the integrator of p; the first `still` bodies do not turn."""
    L, dt, n = p.L, p.dt, x.numel()
    for step in range(steps):
        noise = math.sqrt(2 * p.Dr * dt) * _normal(n, step, 1, p.seed) if p.Dr > 0 else torch.zeros_like(th)
        noise[:still] = 0.0

        def at(h, frac, k):
            return _wrap(x + h * k[0], L), _wrap(y + h * k[1], L), _angle(th + h * k[2] + frac * noise)
        k1 = rates(x, y, th)
        if p.integrator == abi.INT_EULER:
            x, y, th = _wrap(x + dt * k1[0], L), _wrap(y + dt * k1[1], L), th + dt * k1[2] + noise
        elif p.integrator == abi.INT_RK2:
            x, y, th = at(dt, 1.0, rates(*at(dt / 2, 0.5, k1)))
        else:
            k2 = rates(*at(dt / 2, 0.5, k1))
            k3 = rates(*at(dt / 2, 0.5, k2))
            k4 = rates(*at(dt, 1.0, k3))
            x, y, th = at(dt / 6, 1.0, tuple(a + 2 * b + 2 * c + d for a, b, c, d in zip(k1, k2, k3, k4)))
    return x, y, th


def _vicsek64(p, x, y, th, steps):
    L, n = p.L, x.numel()
    for step in range(steps):
        xi = (2.0 * (_words(n, step, 2, p.seed)[0] >> 8).double() * 2.0 ** -24 - 1.0) * math.pi
        i, j = _near(x, y, L, p.r_align)
        if p.model == abi.MODEL_VICSEK:
            sx = torch.cos(th) + _sum(n, i, torch.cos(th[j]))
            sy = torch.sin(th) + _sum(n, i, torch.sin(th[j]))
            th = _angle(torch.atan2(sy, sx) + p.eta * xi)
        elif p.model == abi.MODEL_VICSEK_REF_ANGLE:
            c = _sum(n, i, torch.ones_like(th[j]))
            th = torch.where(c > 0, _sum(n, i, th[j]) / c.clamp(min=1.0), th) + p.eta * xi
        else:
            return None
        x, y = _wrap(x + p.v0 * torch.cos(th), L), _wrap(y + p.v0 * torch.sin(th), L)
    return x, y, th


def _lyapunov64(p, x, y, th, K, steps, every, seed):
    """RK4 of the base system and of its linearisation, QR every `every` steps."""
    n, L, dt = p.n, p.L, p.dt
    near = _Near(L, p.r_align)
    base = _rates_abp(p, near)
    V = torch.stack([torch.stack([_normal(n, 3 * v + c, 5, seed) for c in range(3)]) for v in range(K)])

    def renormalise(V):
        Q, R = torch.linalg.qr(V.reshape(K, -1).T)
        s = torch.sign(torch.diagonal(R))
        return (Q * s).T.reshape(K, 3, n).contiguous(), torch.log(torch.diagonal(R).abs())

    def rates(x, y, th, U):
        i, j = near(x, y)
        dx, dy = _image(x[i] - x[j], L), _image(y[i] - y[j], L)
        al = dx * dx + dy * dy < p.r_align ** 2
        i, j = i[al], j[al]
        c = torch.cos(th[j] - th[i])
        dt_ = torch.stack([_sum(n, i, c * (u[j] - u[i])) for u in U[:, 2]])
        return base(x, y, th) + (torch.stack([-p.v0 * torch.sin(th) * U[:, 2], p.v0 * torch.cos(th) * U[:, 2],
                                              p.g / math.pi * dt_], 1),)

    V, _ = renormalise(V)
    total = torch.zeros(K, dtype=torch.float64, device=DEV)
    for step in range(steps):
        def at(h, k):
            return _wrap(x + h * k[0], L), _wrap(y + h * k[1], L), _angle(th + h * k[2]), V + h * k[3]
        k1 = rates(x, y, th, V)
        k2 = rates(*at(dt / 2, k1))
        k3 = rates(*at(dt / 2, k2))
        k4 = rates(*at(dt, k3))
        x, y, th, V = at(dt / 6, tuple(a + 2 * b + 2 * c + d for a, b, c, d in zip(k1, k2, k3, k4)))
        if (step + 1) % every == 0 or step + 1 == steps:
            V, lr = renormalise(V)
            total += lr
    return total / (steps * dt), V, (x, y, th)


def _fit64(case, d):
    """Adam on FP64 masters; the network reads BF16 copies of them, as the
    surrogate is defined."""
    H, E, B = surrogate.HIDDEN, case["ensemble"], case["samples"]
    T = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=DEV)   # noqa: E731
    x, t, w, th, xq = T(d["x"]), T(d["t"]), T(d["w"]), T(d["theta"]), T(d["xq"])
    w = w / w.sum(1, keepdim=True)
    o1, o2 = H * 7, H * 7 + H
    o3, o4, o5 = o2 + H * H, o2 + H * H + H, o2 + H * H + 2 * H

    def net(q, x):
        W1, b1, W2 = q[:, :o1].view(E, H, 7), q[:, o1:o2], q[:, o2:o3].view(E, H, H)
        b2, W3, b3 = q[:, o3:o4], q[:, o4:o5], q[:, o5:]
        act = lambda z: torch.nn.functional.gelu(z, approximate="tanh")   # noqa: E731
        h = act(torch.einsum("bi,ehi->ebh", x, W1) + b1[:, None])
        h = act(torch.einsum("ebh,egh->ebg", h, W2) + b2[:, None])
        return torch.einsum("ebh,eh->eb", h, W3) + b3

    low = lambda q: q.float().bfloat16().double()   # noqa: E731
    m, v = torch.zeros_like(th), torch.zeros_like(th)
    for it in range(1, case["iters"] + 1):
        q = low(th).requires_grad_(True)
        (w * (net(q, x) - t) ** 2).sum().backward()
        m, v = 0.9 * m + 0.1 * q.grad, 0.999 * v + 0.001 * q.grad ** 2
        th = th - 1e-3 * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
    q = low(th)
    return {"loss": (w * (net(q, x) - t) ** 2).sum(1), "params": th, "y": net(q, xq)}


def exact(case, seed):
    """The same outputs in 64 bits.  None: integer outputs; a running batch
    and Vicsek runs past about ten steps (dt = 1: heading sums that nearly
    cancel turn any rounding into another trajectory); VicsekParticle2."""
    kind = case["kind"]
    if kind in ("series", "sweep", "sweepon", "pairs"):
        return None
    if kind == "fit":
        return _fit64(case, _fit_data(case, seed))
    p = _params(case, seed)
    x, y, th = (torch.tensor(a, dtype=torch.float64, device=DEV) for a in _state(case, p, seed))
    if kind == "lyapunov":
        lam, V, state = _lyapunov64(p, x, y, th, case["k"], case["steps"], case["every"], seed)
        return {"lambda": lam, "span": case["steps"] * p.dt, "vectors": V, "state": state + (None, None)}
    if kind == "vicsek":
        got = _vicsek64(p, x, y, th, case["steps"])
        return None if got is None else {"state": got + (None, None)}
    if kind == "vesicles":
        near = _Near(p.L, p.r_rep)
        got = _advance(p, _rates_vesicles(p, near), x, y, th, case["steps"], still=p.n_rings * p.ring_size)
        return {"state": got + (None, None)}
    near = _Near(p.L, max(p.r_align, p.r_rep))
    steps = case["every"] if kind == "frame" else case["steps"]
    got = _advance(p, _rates_abp(p, near), x, y, th, steps)
    if kind == "frame":
        P = math.hypot(float(torch.cos(got[2]).mean()), float(torch.sin(got[2]).mean()))
        return {"x": got[0], "y": got[1], "theta": got[2], "img_x": None, "img_y": None, "P": P, "step": None}
    return {"state": got + (None, None)}
