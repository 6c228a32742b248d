"""Surrogate-steered parameter sweep.

The reference resolves a sweep by running every point to the end, one
realisation per MPI rank (serial/mpi-main.cpp:157-176).  Here all points run
as one device batch (``Batch``), and an ensemble MLP trained on the sweep's
own completed runs predicts each point's stationary polarization from its
parameters and the moments of its polarization over a short start-up
window.  Points whose predicted error is small retire after the window; the
others run to the end, and a held-out 10% runs to the end to measure the
surrogate's error.

The ensemble is K-fold bagged: member e is fitted with the completed points
of fold e left out (weight 0).  A point's error bound is c x (ensemble
spread), with c a split-conformal multiplier: the ``coverage`` quantile of
|prediction - full run| / spread over the points that were predicted in an
earlier round before they ran; before any such points exist, over the
held-out points, which no fit is trained on (``first_scale="heldout"``;
``"oof"`` takes the out-of-fold multiplier of the fit instead, which runs
about twice as large: a single member's out-of-fold error against the
spread of all five).  A point retires when its bound is at most ``tol``.

Protocol (``run_sweep``):
  1. every point runs ``window`` steps (device-side moments of P);
  2. a pilot subset and the held-out points run to ``max_steps``; their
     stationary P (mean over the second half) are the training targets and
     the held-out points' ground truth;
  3. rounds: fit on all completed non-held-out points; of the points whose
     bound exceeds ``tol``, the ``run_frac`` with the largest bounds (all of
     them in the last round) resume and run to the end -- the plain full run
     is the fallback, and the steps go to the points near the flocking
     transition;
  4. the points left when no bound exceeds ``tol`` retire with the ensemble
     mean of a fit on everything that ran;
  5. the held-out points compare that fit with their full runs.
"""
import ctypes as C
import math
import time
from dataclasses import dataclass, field

import numpy as np

from . import abi, configs
from .system import Batch

HIDDEN = 128
N_FEATURES = 7


def n_params(in_dim=N_FEATURES):
    return HIDDEN * in_dim + HIDDEN + HIDDEN * HIDDEN + HIDDEN + HIDDEN + 1


def init_params(ensemble, in_dim=N_FEATURES, seed=4):
    """Uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases, from
    the Philox stream (member e uses system word e)."""
    P = n_params(in_dim)
    out = np.zeros((ensemble, P), np.float32)
    for e in range(ensemble):
        ids = np.arange(P, dtype=np.uint32)
        u = configs.u01_f32(configs.draw(seed, 100 + e, ids, 0, 8)[0]).astype(np.float64)
        w = 2 * u - 1
        th = np.zeros(P)
        o = 0
        th[o:o + HIDDEN * in_dim] = w[o:o + HIDDEN * in_dim] / math.sqrt(in_dim)
        o = HIDDEN * in_dim + HIDDEN
        th[o:o + HIDDEN * HIDDEN] = w[o:o + HIDDEN * HIDDEN] / math.sqrt(HIDDEN)
        o = HIDDEN * in_dim + HIDDEN + HIDDEN * HIDDEN + HIDDEN
        th[o:o + HIDDEN] = w[o:o + HIDDEN] / math.sqrt(HIDDEN)
        out[e] = th.astype(np.float32)
    return out


class Mlp:
    """Ensemble MLP on the device (spp_mlp_*)."""

    def __init__(self, ensemble=5, in_dim=N_FEATURES, seed=4):
        self._h = C.c_void_p()
        abi.check(abi.lib().spp_mlp_create(ensemble, in_dim, C.byref(self._h)), "spp_mlp_create")
        self.E, self.in_dim = ensemble, in_dim
        self.P = abi.lib().spp_mlp_num_params(self._h)
        self.set_params(init_params(ensemble, in_dim, seed))

    def close(self):
        if self._h:
            abi.lib().spp_mlp_destroy(self._h)
            self._h = C.c_void_p()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def set_params(self, theta):
        theta = np.ascontiguousarray(theta, np.float32).reshape(self.E, self.P)
        abi.check(abi.lib().spp_mlp_set_params(self._h, abi.fptr(theta)), "spp_mlp_set_params")

    def params(self):
        out = np.empty((self.E, self.P), np.float32)
        abi.check(abi.lib().spp_mlp_get_params(self._h, abi.fptr(out)), "spp_mlp_get_params")
        return out

    def predict(self, x):
        x = np.ascontiguousarray(x, np.float32)
        B = x.shape[0]
        y = np.empty((self.E, B), np.float32)
        abi.check(abi.lib().spp_mlp_predict(self._h, abi.fptr(x), B, abi.fptr(y)), "spp_mlp_predict")
        return y

    @staticmethod
    def _weights(w, E, B):
        if w is None:
            return None
        return np.ascontiguousarray(np.broadcast_to(np.asarray(w, np.float32), (E, B)))

    def grad(self, x, t, weights=None):
        """Gradient [E][P] and loss [E] of the weighted squared error
        (weights [E][B] or [B], None = the mean-squared error)."""
        x = np.ascontiguousarray(x, np.float32)
        t = np.ascontiguousarray(t, np.float32)
        w = self._weights(weights, self.E, x.shape[0])
        g = np.empty((self.E, self.P), np.float32)
        loss = np.empty(self.E, np.float32)
        abi.check(abi.lib().spp_mlp_grad(self._h, abi.fptr(x), abi.fptr(t), abi.fptr(w), x.shape[0],
                                         abi.fptr(g), abi.fptr(loss)), "spp_mlp_grad")
        return g, loss

    def resident_launches(self):
        """Launches so far that ran many training iterations each."""
        return int(abi.lib().spp_mlp_resident_launches(self._h))

    def train(self, x, t, iters=2000, lr=1e-3, weights=None):
        x = np.ascontiguousarray(x, np.float32)
        t = np.ascontiguousarray(t, np.float32)
        w = self._weights(weights, self.E, x.shape[0])
        loss = np.empty(self.E, np.float32)
        abi.check(abi.lib().spp_mlp_train(self._h, abi.fptr(x), abi.fptr(t), abi.fptr(w), x.shape[0],
                                          int(iters), float(lr), abi.fptr(loss)), "spp_mlp_train")
        return loss


def features(points, stats):
    """(eta, rho, v0, log N, mean P, log var P, log kurtosis P) per point,
    the moments over the start-up window.  Variance and kurtosis span
    decades across a sweep, so they enter as logarithms."""
    f = np.zeros((len(points), N_FEATURES))
    for s, (p, st) in enumerate(zip(points, stats)):
        rho = p.n / (4.0 * p.L * p.L)
        f[s] = [p.eta, rho, p.v0, math.log(p.n), st.p_mean, math.log(max(st.p_var, 0.0) + 1e-8),
                math.log(max(st.p_kurt, 0.0) + 1e-8)]
    return f


def kfold(n, k, seed):
    """Fold index of each of n samples: a seeded permutation dealt into k folds."""
    fold = np.empty(n, np.int64)
    fold[np.random.default_rng(seed).permutation(n)] = np.arange(n) % k
    return fold


@dataclass
class Surrogate:
    """K-fold bagged ensemble with a conformal error bound (module docstring)."""
    ensemble: int = 5
    seed: int = 4
    iters: int = 3000
    lr: float = 1e-3
    coverage: float = 0.8
    spread_floor: float = 1e-3
    mu: np.ndarray = field(default=None)
    sd: np.ndarray = field(default=None)
    oof_scale: float = math.inf
    loss: np.ndarray = field(default=None)
    mlp: Mlp = field(default=None)

    def _norm(self, f):
        return ((f - self.mu) / self.sd).astype(np.float32)

    def fit(self, f, target):
        """Fits member e with fold e of the samples left out and sets
        oof_scale, the coverage quantile of |out-of-fold error| / spread."""
        f = np.asarray(f, np.float64)
        target = np.asarray(target, np.float64)
        n, E = len(target), self.ensemble
        self.mu = f.mean(0)
        self.sd = f.std(0) + 1e-9
        if self.mlp is None:
            self.mlp = Mlp(E, f.shape[1], self.seed)
        else:
            self.mlp.set_params(init_params(E, f.shape[1], self.seed))
        fold = kfold(n, E, self.seed)
        w = (fold[None, :] != np.arange(E)[:, None]).astype(np.float32)
        if n < 2 * E:
            w[:] = 1.0  # too few points to leave folds out: plain ensemble, no bound
        self.loss = self.mlp.train(self._norm(f), target.astype(np.float32), self.iters, self.lr, weights=w)
        if n < 2 * E:
            self.oof_scale = math.inf
            return self.loss
        y = self.mlp.predict(self._norm(f)).astype(np.float64)
        oof = y[fold, np.arange(n)]
        self.oof_scale = float(np.quantile(np.abs(oof - target) / self.floor(y.std(0)), self.coverage))
        return self.loss

    def floor(self, spread):
        return np.maximum(spread, self.spread_floor)

    def predict(self, f):
        """(ensemble mean, ensemble spread) per row of f."""
        y = self.mlp.predict(self._norm(np.asarray(f, np.float64))).astype(np.float64)
        return y.mean(0), y.std(0)


@dataclass
class SweepResult:
    p_answer: np.ndarray          # stationary P reported per point
    p_full: np.ndarray            # P of the points run to the end (NaN otherwise)
    bound: np.ndarray             # error bound of the decision that retired a point (NaN otherwise)
    retired: np.ndarray           # bool: answered by the surrogate
    heldout: np.ndarray           # bool: held-out points (always run in full)
    heldout_err: np.ndarray       # |prediction - full run| on the held-out points
    particle_steps: int           # work actually done
    particle_steps_plain: int     # work of running every point to the end
    rounds: int
    scales: list                  # conformal multiplier of each round
    wall_s: float
    timings: dict


def pilot_points(points, candidates, count, how, seed):
    """The pilot subset: `count` of the `candidates` (indices).  how="random":
    a seeded random draw.  how="cheap": the parameter plane (eta, rho) is cut
    into a 6 x 6 grid of strata, and each stratum gives its smallest systems
    in proportion to its share of the candidates, so the pilot still covers
    the plane while its full runs, which every later decision waits for,
    take a small share of the particle-steps."""
    candidates = np.asarray(candidates)
    if how == "random":
        return np.random.default_rng(seed).permutation(candidates)[:count]
    eta = np.array([points[i].eta for i in candidates])
    rho = np.array([points[i].n / (4.0 * points[i].L * points[i].L) for i in candidates])
    size = np.array([points[i].n for i in candidates])
    def cut(v):
        edges = np.quantile(v, np.linspace(0, 1, 7)[1:-1])
        return np.searchsorted(edges, v, side="right")
    stratum = cut(eta) * 6 + cut(rho)
    picked = []
    frac = count / len(candidates)
    for s_ in np.unique(stratum):
        members = np.flatnonzero(stratum == s_)
        members = members[np.argsort(size[members], kind="stable")]
        picked.extend(members[:max(1, int(round(frac * len(members))))].tolist())
    picked = np.array(picked)
    if len(picked) > count:   # rounding: drop the largest
        picked = picked[np.argsort(size[picked], kind="stable")][:count]
    return candidates[picked]


def run_sweep(points, max_steps=20000, window=500, pilot_frac=0.2, holdout_frac=0.1, tol=0.02,
              max_rounds=1, run_frac=0.5, surrogate=None, seed=4, x0=None, use_surrogate=True,
              chunk=2000, exchange=None, pilot_select="random", speculate_frac=0.0,
              first_scale="heldout"):
    """Runs the sweep and returns a SweepResult.  With use_surrogate=False
    every point runs to the end (the plain batched sweep).

    exchange (spp_gb300.replicas.Exchange) makes this one shard of a sweep
    over several ranks: every fit uses all ranks' completed points, the
    conformal multiplier all ranks' fresh residuals, and the rounds end
    together (their collectives stay matched); without it the sweep is
    local.

    Rounds r = 0 .. max_rounds: fit on every completed non-held-out point;
    the error bound of a remaining point is c x spread, with c the coverage
    quantile of |prediction - full run| / spread over the points predicted
    in earlier rounds before they ran (split conformal on fresh residuals;
    before any exist, on the held-out points or, with first_scale="oof",
    the out-of-fold multiplier).  Measured on the 512-point workload (one
    GB300, points/hour at |dP| <= 0.02 against the plain batched sweep, with
    batch kernels that took 16.8 s for it, now 10.0), coverage 0.9: held-out first scale with one round 1.07x, with two rounds
    1.01x; out-of-fold first scale with two rounds 1.03x.  The coverage
    trades retirements for accuracy (held-out first scale, one round):
    0.9 -> 1.07x, 98.3% of the retired points within tolerance; 0.8 (the
    default) -> 1.15x, 96.2%; 0.7 -> 1.22x, 94.3%.  Of the
    points whose bound exceeds tol, the run_frac with the largest bounds run
    to the end (all of them in the last round); the points left when no
    bound exceeds tol retire with the mean of a fit on everything run."""
    from .replicas import Exchange
    ex = exchange if exchange is not None else Exchange()
    t_start = time.perf_counter()
    timings = {"runs_s": 0.0, "train_s": 0.0}
    n = len(points)
    rng = np.random.default_rng(seed)
    order = rng.permutation(n)
    n_hold = max(1, int(round(holdout_frac * n)))
    heldout = np.zeros(n, bool)
    heldout[order[:n_hold]] = True
    pilot = np.zeros(n, bool)
    n_pilot = max(2, int(round(pilot_frac * n)))
    if pilot_select == "random":
        pilot[order[n_hold:n_hold + n_pilot]] = True
    else:
        pilot[pilot_points(points, order[n_hold:], n_pilot, pilot_select, seed)] = True
    stationary_from = max_steps // 2
    x, y, th = x0 if x0 is not None else configs.sweep_state(points, seed=seed)
    sizes = np.array([p.n for p in points], np.int64)
    retired = np.zeros(n, bool)
    bound = np.full(n, np.nan)
    heldout_err = np.array([])
    rounds, scales = 0, []
    with Batch(points) as b:
        b.set_windows(window, stationary_from, max_steps)
        b.upload(x, y, th)

        timings["phases"] = []

        def run(systems=None):
            t0 = time.perf_counter()
            if systems is not None:
                resume(b, systems)
            act = np.array([s.active for s in b.poll()], bool)
            run_until_done(b, chunk)
            dt_ = time.perf_counter() - t0
            timings["runs_s"] += dt_
            timings["phases"].append({"points": int(act.sum()), "particles": int(sizes[act].sum()),
                                      "wall_s": dt_})

        if use_surrogate:
            t0 = time.perf_counter()
            b.step(window)
            timings["runs_s"] += time.perf_counter() - t0
            f = features(points, b.poll())
            if speculate_frac > 0:
                # points likely to stay unsure (the largest start-up-window
                # variance of P: fluctuating, near the transition) run to the
                # end with the pilot and join its training data
                cand = np.flatnonzero(~(pilot | heldout))
                k_spec = int(round(speculate_frac * n))
                spec = cand[np.argsort(-f[cand, 5], kind="stable")][:k_spec]
                pilot[spec] = True
            # only the pilot and held-out points continue for now
            b.retire(np.flatnonzero(~(pilot | heldout)))
        run()
        st = b.poll()
        p_full = np.array([s.p_stationary if s.steps >= max_steps else np.nan for s in st])
        if use_surrogate:
            sur = surrogate or Surrogate(seed=seed)
            remaining = ~(pilot | heldout)
            fresh = []
            for r in range(max_rounds + 2):
                t1 = time.perf_counter()
                done = np.isfinite(p_full) & ~heldout
                f_fit, p_fit = ex([f[done], p_full[done]])
                sur.fit(f_fit, p_fit)
                mean, spread = sur.predict(f)
                timings["train_s"] += time.perf_counter() - t1
                if r == max_rounds + 1 or not ex.any(remaining.any()):
                    break
                rounds += 1
                res_all = ex([np.concatenate(fresh) if fresh else np.zeros(0)])[0]
                if res_all.size:
                    scale = float(np.quantile(res_all, sur.coverage))
                elif first_scale == "heldout":
                    # split conformal on the held-out points, which no fit has
                    # seen: their residuals under this fit calibrate the bound
                    h = np.flatnonzero(heldout)
                    res_h = ex([np.abs(mean[h] - p_full[h]) / sur.floor(spread[h])])[0]
                    scale = float(np.quantile(res_h, sur.coverage))
                else:
                    scale = sur.oof_scale
                scales.append(scale)
                bnd = scale * sur.floor(spread)
                bound[remaining] = bnd[remaining]
                unsure = np.flatnonzero(remaining & (bnd > tol))
                if not ex.any(unsure.size > 0):
                    break
                if r < max_rounds and unsure.size:
                    keep = max(1, int(math.ceil(run_frac * unsure.size)))
                    unsure = unsure[np.argsort(-bnd[unsure], kind="stable")][:keep]
                if unsure.size:
                    run(unsure)
                st = b.poll()
                for s in unsure:
                    p_full[s] = st[s].p_stationary
                fresh.append(np.abs(mean[unsure] - p_full[unsure]) / sur.floor(spread[unsure]))
                remaining[unsure] = False
                bound[unsure] = np.nan
            retired = remaining
            heldout_err = np.abs(mean[heldout] - p_full[heldout])
        p_answer = np.where(retired, mean, p_full) if use_surrogate else p_full.copy()
        steps = np.array([s.steps for s in b.poll()], np.int64)
        wall = time.perf_counter() - t_start
    return SweepResult(p_answer=p_answer, p_full=p_full, bound=bound, retired=retired, heldout=heldout,
                       heldout_err=heldout_err, particle_steps=int(np.sum(sizes * steps)),
                       particle_steps_plain=int(np.sum(sizes) * max_steps), rounds=rounds, scales=scales,
                       wall_s=wall, timings=timings)


def run_until_done(b, chunk):
    while True:
        st = b.poll()
        if not any(s.active for s in st):
            return
        b.step(chunk)


def resume(b, systems):
    b.resume(systems)
