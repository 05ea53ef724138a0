"""The workloads that performance work on the tracer is measured on.

Every case is one advance of an ensemble of tracers through the package's
public entry points, as a user's program makes it: the start state goes from
host memory to the device, the ensemble advances, and the tracers' states (and,
where the program wants the trajectories, their output rows) come back. The
start state is kept apart, so that every pass starts from it.

Families (``listed()`` says what each case stands for, ``draw()`` spreads the
sizes and options of the same families):

  gc         guiding centres in the double dipole (config 2's electrons)
  particles  full orbits in the Earth dipole
  adaptive   the particle / guiding-centre switch, Harris sheet or breathing dipole
  grid       guiding centres in a gridded field
  bounce     guiding centres at the reference's default cadence, a tenth of the
             bounce period
  bc         bounce centres (BounceCenter)

Durations stop short of where rounding alone moves a trajectory visibly: 50
gyro-periods of a nonadiabatic proton, or seconds of a guiding centre between
the cells of a linearly interpolated field, are chaotic.

``exact`` restates the same integrations in 64-bit torch: the equations of
motion, the Dormand-Prince pairs with Hairer's step-size control restarted at
every output row, the adaptive switch, the field-line traces with their
quadratic splines.
"""
import math

import numpy as np
import torch

from rapt_gb300 import _native as N
from rapt_gb300 import fields as F
from rapt_gb300 import learned
from rapt_gb300 import workloads as W
from rapt_gb300.ensemble import Ensemble

RE, B0, C, QE, ME, MP = W.Re, W.B0, W.c, W.e, W.m_el, W.m_pr
PLAIN, FP32, LEARNED_FP32 = 0, 1, 3


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one guiding centre and its trajectory: the reference's own unit of work (GuidingCenter.advance)
        {"name": "gc_one", "family": "gc", "n": 1, "form": PLAIN, "dense": False, "delta": 1.0, "cadence": 0.1,
         "rows": True},
        # a plain FP64 ensemble at config 2's size (65,536 electrons)
        {"name": "gc_64k", "family": "gc", "n": 65536, "form": PLAIN, "dense": False, "delta": 0.5, "cadence": 0.5,
         "rows": False},
        # trajectories on a fine cadence through dense output (odd size)
        {"name": "gc_dense_rows", "family": "gc", "n": 10007, "form": PLAIN, "dense": True, "delta": 0.25,
         "cadence": 0.01, "rows": True},
        # the FP32 form without the network
        {"name": "gc_fp32_256k", "family": "gc", "n": 262144, "form": FP32, "dense": False, "delta": 0.5,
         "cadence": 0.5, "rows": False},
        # the headline: 2^20 electrons, learned + FP32, one 1 s step
        {"name": "gc_learned_1m", "family": "gc", "n": 1048576, "form": LEARNED_FP32, "dense": False, "delta": 1.0,
         "cadence": 1.0, "rows": False},
        # config 1: 256 protons from 6 Re with their trajectories, 20 rows a gyration
        {"name": "particles_256", "family": "particles", "n": 256, "form": PLAIN, "mixed": False, "span": 1.0,
         "resolution": 20, "rows": True},
        # config 4's mixed species as a trapped population, 8 gyro-periods
        {"name": "particles_200k", "family": "particles", "n": 200000, "form": PLAIN, "mixed": True, "span": 8.05,
         "resolution": 10, "rows": False},
        # config 3: protons in the Harris sheet, uneven durations
        {"name": "harris_32k", "family": "adaptive", "field": "Harris", "n": 32768, "delta": 20.0, "cadence": 0.5},
        # config 5: mixed species in the breathing dipole
        {"name": "compressed_3k", "family": "adaptive", "field": "CompressedDipole", "n": 3001, "delta": 0.5,
         "cadence": 0.25},
        # gridded fields as an MHD code writes them, time dependent, with E
        {"name": "grid_16k", "family": "grid", "n": 16384, "nodes": 121, "delta": 0.25},
        # the reference's default cadence (GCtimestep = 0): the bounce period first, then a row every tenth of it
        {"name": "bounce_16k", "family": "bounce", "n": 16384, "delta": 0.2, "resolution": 10},
        # bounce centres: five field-line traces per right-hand side
        {"name": "bc_2k", "family": "bc", "n": 2048, "delta": 0.2},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    family = rng.choice(["gc", "gc", "particles", "adaptive", "grid", "bounce", "bc"])
    if family == "gc":
        form = rng.choice([PLAIN, PLAIN, PLAIN, FP32, LEARNED_FP32])
        dense = form == PLAIN and rng.random() < 0.3
        n = _spread(rng, 1, {PLAIN: 65536, FP32: 262144, LEARNED_FP32: 1048576}[form] // (4 if dense else 1))
        delta = rng.uniform(0.1, 0.5)
        return {"family": "gc", "n": n, "form": form, "dense": dense, "delta": delta,
                "cadence": 0.01 if dense else delta / rng.randint(1, 4), "rows": n <= 10007}
    if family == "particles":
        mixed = rng.random() < 0.6
        n = _spread(rng, 1, 200000 if mixed else 4096)
        return {"family": "particles", "n": n, "form": rng.choice([PLAIN, PLAIN, FP32]), "mixed": mixed,
                "span": rng.randint(3, 7) + 0.05 if mixed else rng.uniform(0.5, 1.0),
                "resolution": rng.choice([10, 20]), "rows": not mixed}
    if family == "adaptive":
        if rng.random() < 0.6:
            return {"family": "adaptive", "field": "Harris", "n": _spread(rng, 1, 32768),
                    "delta": rng.uniform(2.0, 20.0), "cadence": 0.5}
        return {"family": "adaptive", "field": "CompressedDipole", "n": _spread(rng, 1, 3001),
                "delta": rng.uniform(0.2, 0.5), "cadence": rng.uniform(0.1, 0.3)}
    if family == "grid":
        return {"family": "grid", "n": _spread(rng, 1, 16384), "nodes": rng.randrange(61, 122, 4),
                "delta": rng.uniform(0.1, 0.25)}
    if family == "bounce":
        return {"family": "bounce", "n": _spread(rng, 1, 16384), "delta": rng.uniform(0.05, 0.2),
                "resolution": rng.randint(9, 11)}
    return {"family": "bc", "n": _spread(rng, 1, 2048), "delta": rng.uniform(0.05, 0.2)}


# ------------------------------------------------------------------ inputs
def _trapped(n, seed):
    """Protons and electrons, half each: L 3-6 in the equator, 10 keV-1 MeV, pitch angle 30-85 degrees."""
    rng = np.random.default_rng(seed)
    pos = W._equatorial(rng, n, 3.0, 6.0)
    ke = 10 ** rng.uniform(4, 6, n)
    alpha, phase = np.deg2rad(rng.uniform(30, 85, n)), rng.uniform(0, 2 * np.pi, n)
    electron = np.arange(n) % 2 == 1
    mass, charge = np.where(electron, ME, MP), np.where(electron, -QE, QE)
    v = W.speed_from_ke(ke, mass)
    period = 2 * np.pi * mass / np.sqrt(1 - (v / C) ** 2) / (B0 * RE ** 3 / np.linalg.norm(pos, axis=1) ** 3 * QE)
    return {"pos": pos, "vel": W._velocity(W._dipole_bhat(pos), v, alpha, phase), "mass": mass, "charge": charge,
            "period": period}


def _workload(case, seed):
    """(workload, kind, delta): initial states by species, position and velocity, and the duration of the advance."""
    fam, n = case["family"], case["n"]
    if fam == "gc":
        w = W.config2(n, seed)
        w["params"] = dict(rtol=1e-8, atol=1e-8, gctimestep=case["cadence"], form=case["form"],
                           dense_output=int(case["dense"]))
        return w, "gc", case["delta"]
    if fam == "particles":
        w = W.config1(n, seed)
        w["params"] = dict(rtol=1e-8, atol=1e-8, cyclotronresolution=case["resolution"], form=case["form"])
        if not case["mixed"]:
            return w, "particle", case["span"]
        w.update(_trapped(n, seed))
        return w, "particle", case["span"] * w["period"]
    if fam == "adaptive":
        if case["field"] == "Harris":
            w = W.config3(n, seed)
            delta = case["delta"] * 10 ** np.random.default_rng(seed + 1).uniform(-1, 0, n)
        else:
            w = W.config5(n, seed)
            delta = np.full(n, case["delta"])
        w["params"] = dict(rtol=1e-8, atol=1e-8, gctimestep=case["cadence"])
        return w, "adaptive", delta
    if fam == "grid":
        w = W.config2(n, seed)
        w["params"] = dict(rtol=1e-6, atol=1e-6, gctimestep=case["delta"])
        return w, "gc", case["delta"]
    if fam == "bounce":
        w = W.config2(n, seed)
        w["params"] = dict(rtol=1.49012e-8, atol=1.49012e-8, gctimestep=0.0, bounceresolution=case["resolution"])
        return w, "gc", case["delta"]
    return W.bc_drift(n, seed), "bc", case["delta"]


_grid = None


def _dipole_grid(nodes):
    """The gridded dipole with E (workloads.dipole_grid), its last one kept: it does not depend on the seed."""
    global _grid
    if _grid is None or _grid[0] != nodes:
        _grid = (nodes, W.dipole_grid(nodes, nodes, nodes // 2 + 1))
    return _grid[1]


def _field(case, w):
    return _dipole_grid(case["nodes"]) if case["family"] == "grid" else getattr(F, w["field"][0])(**w["field"][1])


def _wants_rows(case):
    return case.get("rows", False) or case["n"] <= 4096 and (case["family"] == "bounce" or case.get("field") == "Harris")


def _max_rows(case):
    """Row capacity: a few where only the final state is read, all rows where the trajectories are."""
    fam = case["family"]
    if fam == "gc":
        return int(math.ceil(case["delta"] / case["cadence"])) + (20 if case["dense"] else 3)
    if fam == "particles":
        return 256 if case["rows"] else int(case["resolution"] * (case["span"] + 2))
    if fam == "adaptive":
        return 512 if case["field"] == "Harris" else 16384
    return 128 if fam == "bounce" else 4


def _train(ctx, seed):
    """The step network of the learned form, trained on electrons of the same distributions."""
    return learned.fit_gc(W.config2(512, seed + 7), 1.0, ctx=ctx, rounds=1, steps=400, batch=1024, capacity=1 << 18,
                          seed=seed)[0]


def prepare(case, seed):
    w, kind, delta = _workload(case, seed)
    ctx = N.Context()
    if kind == "bc":
        gamma = 1 / np.sqrt(1 - (w["v"] / C) ** 2)
        field = _field(case, w)
        pts = np.column_stack([np.zeros(case["n"]), w["pos"]])
        mu = (gamma * w["v"] * np.sin(np.deg2rad(w["eqpa"]))) ** 2 * w["mass"] / (2 * field.magB(pts))
        p = w["params"]
        field.bind(ctx)
        ctx.set_config(rtol=p["rtol"], atol=p["atol"])
        return {"kind": kind, "ctx": ctx, "delta": delta, "state": np.column_stack([pts, np.zeros(case["n"])]),
                "cst": np.column_stack([w["v"], mu, w["mass"], w["charge"]]), "params": p}
    learn = case.get("form") == LEARNED_FP32
    if learn:
        net = _train(ctx, seed)
    ens = Ensemble(_field(case, w), case["n"], max_rows=_max_rows(case), ctx=ctx,
                   max_switch=8 if kind == "adaptive" else 0)
    if learn:
        ctx.mlp_set_params(net)
    ens.configure(**w["params"], **({"learned_every": 4, "learned_scale": 0.75} if learn else {}))
    if kind == "gc":
        ens.set_guiding_centers(w["pos"], w["v"], pa=w["pa"], t0=0.5 if case["family"] == "grid" else 0.0,
                                mass=w["mass"], charge=w["charge"])
    else:
        ens.set_particles(w["pos"], w["vel"], 0.0, w["mass"], w["charge"])
    start = ens.h
    ens.pin()
    ens.h = {k: np.zeros_like(v) for k, v in start.items()}
    ens.pin()
    return {"kind": kind, "ens": ens, "delta": delta, "start": start, "result": ens.h,
            "rows": _wants_rows(case)}


def run(state):
    if state["kind"] == "bc":
        p = state["params"]
        st, rows, nrows, status, _ = state["ctx"].bc_advance(state["state"].copy(), state["cst"], state["delta"],
                                                             p["bctimestep"], p["eyegradientstep"], 16)
        rows = np.where(np.arange(16)[None, :, None] < nrows[:, None, None], rows, 0.0)
        return {"state": st, "rows": rows, "nrows": nrows, "status": status}
    ens = state["ens"]
    ens.h = state["start"]
    ens.upload()
    if state["kind"] == "adaptive":
        ens.adaptive_init()
    ens.advance(state["kind"], state["delta"])
    ens.h = state["result"]
    h = ens.download()
    out = {"pos": h["s"][:3], "mom": h["s"][3:], "t": h["t_row"], "mode": h["mode"], "status": h["status"]}
    if state["kind"] == "adaptive":
        out["mu"] = h["mu"]
    if state["rows"]:
        rows, _, nrows, _, _ = ens.rows()
        out["rows"] = np.where(np.arange(rows.shape[1])[None, :, None] < nrows[:, None, None], rows, 0.0)
        out["nrows"] = nrows
    return out


def work(case):
    """State in and out (16 and 13 words a tracer), the rows wanted, and the field arithmetic of the steps that the
    tolerance asks for (mean step counts of these distributions; FMA = 2, a division or square root 1)."""
    n, fam = case["n"], case["family"]
    words, rows = 29.0, 0.0
    if fam == "gc":
        # 153 steps a simulated second at rtol 1e-8, 3,093 flops each
        flops = n * case["delta"] * 153.0 * 3093.0
        rows = case["delta"] / case["cadence"] if case["rows"] else 0.0
    elif fam == "particles":
        # 2 DOP853 steps an output interval (0.7 s a gyration at 6 Re): 12 right-hand sides of 45 flops and ~1,100
        # flops of stage sums and error norms
        turns = case["span"] * (1.0 if case["mixed"] else 2.0)
        flops = n * turns * case["resolution"] * 2.0 * 1640.0
        rows = turns * case["resolution"] if case["rows"] else 0.0
    elif fam == "adaptive":
        # about 8 steps a second in the sheet (mean duration 0.39 of the longest), 300 in the breathing dipole
        harris = case["field"] == "Harris"
        flops = n * case["delta"] * (0.39 * 8.0 * 1800.0 if harris else 300.0 * 3000.0)
        rows = case["delta"] if _wants_rows(case) else 0.0
    elif fam == "grid":
        flops = n * case["delta"] * 190.0 * 10200.0
        return {"bytes": 8.0 * (words * n + 18.0 * case["nodes"] ** 2 * (case["nodes"] // 2 + 1)), "flops": flops}
    elif fam == "bounce":
        # the steps, and one field-line trace: ~200 points of 6 field values (~50 flops) and the panel integrals
        flops = n * (case["delta"] * 170.0 * 3093.0 + 200.0 * (6 * 50.0 + 200.0))
        rows = 8.0 if _wants_rows(case) else 0.0
    else:
        # five traces of ~60 points a right-hand side, ~20 right-hand sides a row, about two rows
        flops = n * (1.0 + case["delta"]) * 20.0 * 5.0 * 60.0 * 500.0
        words, rows = 17.0, 1.0 + case["delta"]
    return {"bytes": 8.0 * n * (words + 7.0 * rows), "flops": flops}


# ------------------------------------------------------------------ the same integrations in 64-bit torch
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _T(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device=_dev())


def _dipole(x, y, z):
    """The Earth's dipole: (B0 Re^3 / r^5) (-3xz, -3yz, x^2 + y^2 - 2 z^2)."""
    r2 = x * x + y * y + z * z
    s = -B0 * RE ** 3 / (r2 * r2 * torch.sqrt(r2))
    return torch.stack([3 * x * z * s, 3 * y * z * s, (2 * z * z - x * x - y * y) * s])


class _Model:
    """B(t, X), E(t, X) for X[3, n], with the steps of the central differences."""
    static, gradstep, timestep = True, RE / 1000, 1e-3

    def E(self, t, X):
        return torch.zeros_like(X)


class _Earth(_Model):
    gradstep = RE * 1e-6

    def B(self, t, X):
        return _dipole(X[0], X[1], X[2])


class _Double(_Model):
    def B(self, t, X):
        return _dipole(X[0], X[1], X[2]) + _dipole(X[0] - 20 * RE, X[1], X[2])


class _Harris(_Model):
    static, gradstep = False, 0.5 * RE * 1e-4

    def B(self, t, X):
        z = X[2]
        return torch.stack([20e-9 * torch.tanh(z / (0.5 * RE)), torch.zeros_like(z), torch.full_like(z, 2e-9)])

    def E(self, t, X):
        z = X[2]
        return torch.stack([torch.zeros_like(z), torch.full_like(z, 0.2e-3), torch.zeros_like(z)])


class _Breathing(_Model):
    static = False
    amp, w = 0.1, 2 * np.pi / 60.0

    def B(self, t, X):
        return _dipole(X[0], X[1], X[2]) * (1 + self.amp * torch.sin(self.w * t))

    def E(self, t, X):
        x, y, z = X
        s = -B0 * self.amp * self.w * RE ** 3 * torch.cos(self.w * t) / (x * x + y * y + z * z) ** 1.5
        return torch.stack([s * y, -s * x, torch.zeros_like(x)])


class _Gridded(_Model):
    """Linear interpolation over (t, x, y, z)."""
    static, gradstep = False, 1e-3 * RE

    def __init__(self, g):
        self.ax = [_T(a) for a in (g._t, g._x, g._y, g._z)]
        self.V = torch.cat([_T(g._B), _T(g._E)], dim=-1)

    def _at(self, t, X, lo, hi):
        cell, w = [], []
        for a, v in zip(self.ax, (t, X[0], X[1], X[2])):
            v = v.contiguous()
            i = torch.clamp(torch.searchsorted(a, v, right=True) - 1, 0, len(a) - 2)
            cell.append(i)
            w.append((v - a[i]) / (a[i + 1] - a[i]))
        out = 0.0
        for k in range(16):
            b = [(k >> 3) & 1, (k >> 2) & 1, (k >> 1) & 1, k & 1]
            f = 1.0
            for j in range(4):
                f = f * (w[j] if b[j] else 1 - w[j])
            out = out + self.V[cell[0] + b[0], cell[1] + b[1], cell[2] + b[2], cell[3] + b[3], lo:hi] * f[:, None]
        return out.T

    def B(self, t, X):
        return self._at(t, X, 0, 3)

    def E(self, t, X):
        return self._at(t, X, 3, 6)


def _unit(m, t, X):
    b = m.B(t, X)
    mag = torch.sqrt((b * b).sum(0))
    return b / mag, mag


def _shift(X, a, d):
    Y = X.clone()
    Y[a] += d
    return Y


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _around(m, t, X, times=False):
    """B at X, at X +- d e_a for the central differences in space, and (times) at t -+ the time step: [3, 7 or 9, n]."""
    d, e = m.gradstep, m.timestep
    P = [X] + [_shift(X, a, s) for a in range(3) for s in (d, -d)] + ([X, X] if times else [])
    T = [t] * 7 + ([t - e, t + e] if times else [])
    return m.B(torch.cat(T), torch.cat(P, dim=1)).reshape(3, len(P), -1)


def _gc_rhs(m):
    """The Tao-Chan-Brizard equations with the field's central differences; consts (q, mu, mass)."""
    def f(t, y, c):
        X, pp = y[:3], y[3]
        q, mu, mass = c[0], c[1], c[2]
        Bs = _around(m, t, X, not m.static)
        mags = torch.sqrt((Bs * Bs).sum(0))
        us = Bs / mags
        B, b, mag, d = Bs[:, 0], us[:, 0], mags[0], m.gradstep
        gB = torch.stack([(mags[1 + 2 * a] - mags[2 + 2 * a]) / (2 * d) for a in range(3)])
        D = [(us[:, 1 + 2 * a] - us[:, 2 + 2 * a]) / (2 * d) for a in range(3)]
        curl = torch.stack([D[1][2] - D[2][1], D[2][0] - D[0][2], D[0][1] - D[1][0]])
        db = 0.0 if m.static else (us[:, 8] - us[:, 7]) / (2 * m.timestep)
        gam = torch.sqrt(1 + 2 * mu * mag / (mass * C * C) + (pp / (mass * C)) ** 2)
        Bs = B + pp / q * curl
        par = (Bs * b).sum(0)
        Es = m.E(t, X) - (pp * db + mu / gam * gB) / q
        v = (pp / (gam * mass) * Bs + _cross(Es, b)) / par
        return torch.cat([v, (q * (Es * Bs).sum(0) / par)[None]])
    return f


def _particle_rhs(m):
    """Newton-Lorentz; consts (q, mass, gamma mass at the start of the advance: frozen in static fields)."""
    def f(t, y, c):
        X, p = y[:3], y[3:]
        gm = c[2] if m.static else torch.sqrt(c[1] ** 2 + (p * p).sum(0) / C ** 2)
        return torch.cat([p / gm, c[0] * (m.E(t, X) + _cross(p / gm, m.B(t, X)))])
    return f


# Dormand and Prince's pairs: rows of the tableau, nodes, and the error weights
_A5 = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
       [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
       [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_C5 = [1 / 5, 3 / 10, 4 / 5, 8 / 9, 1, 1]
_E5 = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]
_D5 = [-12715105075 / 11282082432, 0, 87487479700 / 32700410799, -10690763975 / 1880347072,
       701980252875 / 199316789632, -1453857185 / 822651844, 69997945 / 29380423]
_A8 = [[5.26001519587677318785587544488e-2], [1.97250569845378994544595329183e-2, 5.91751709536136983633785987549e-2],
       [2.95875854768068491816892993775e-2, 0, 8.87627564304205475450678981324e-2],
       [2.41365134159266685502369798665e-1, 0, -8.84549479328286085344864962717e-1, 9.24834003261792003115737966543e-1],
       [3.7037037037037037037037037037e-2, 0, 0, 1.70828608729473871279604482173e-1, 1.25467687566822425016691814123e-1],
       [3.7109375e-2, 0, 0, 1.70252211019544039314978060272e-1, 6.02165389804559606850219397283e-2, -1.7578125e-2],
       [3.70920001185047927108779319836e-2, 0, 0, 1.70383925712239993810214054705e-1, 1.07262030446373284651809199168e-1,
        -1.53194377486244017527936158236e-2, 8.27378916381402288758473766002e-3],
       [6.24110958716075717114429577812e-1, 0, 0, -3.36089262944694129406857109825, -8.68219346841726006818189891453e-1,
        2.75920996994467083049415600797e1, 2.01540675504778934086186788979e1, -4.34898841810699588477366255144e1],
       [4.77662536438264365890433908527e-1, 0, 0, -2.48811461997166764192642586468, -5.90290826836842996371446475743e-1,
        2.12300514481811942347288949897e1, 1.52792336328824235832596922938e1, -3.32882109689848629194453265587e1,
        -2.03312017085086261358222928593e-2],
       [-9.3714243008598732571704021658e-1, 0, 0, 5.18637242884406370830023853209, 1.09143734899672957818500254654,
        -8.14978701074692612513997267357, -1.85200656599969598641566180701e1, 2.27394870993505042818970056734e1,
        2.49360555267965238987089396762, -3.0467644718982195003823669022],
       [2.27331014751653820792359768449, 0, 0, -1.05344954667372501984066689879e1, -2.00087205822486249909675718444,
        -1.79589318631187989172765950534e1, 2.79488845294199600508499808837e1, -2.85899827713502369474065508674,
        -8.87285693353062954433549289258, 1.23605671757943030647266201528e1, 6.43392746015763530355970484046e-1],
       [5.42937341171687622380535766363e-2, 0, 0, 0, 0, 4.45031289275240888144113950566,
        1.89151789931450038304281599044, -5.8012039600105847814672114227, 3.1116436695781989441890606237e-1,
        -1.52160949662516078556178806805e-1, 2.01365400804030348374776537501e-1, 4.47106157277725905176885569043e-2]]
_C8 = [.526001519587677318785587544488e-1, .789002279381515978178381316732e-1, .118350341907227396726757197510,
       .281649658092772603273242802490, 1 / 3, .25, 4 / 13, .651282051282051282051282051282, .6,
       .857142857142857142857142857142, 1]
_E8 = [.1312004499419488073250102996e-1, 0, 0, 0, 0, -.1225156446376204440720569753e1, -.4957589496572501915214079952,
       .1664377182454986536961530415e1, -.3503288487499736816886487290, .3341791187130174790297318841,
       .8192320648511571246570742613e-1, -.2235530786388629525884427845e-1]
_B3 = {0: .244094488188976377952755905512, 8: .733846688281611857341361741547, 11: .220588235294117647058823529412e-1}


def _sum(w, k):
    out = 0.0
    for a, v in zip(w, k):
        if a:
            out = out + a * v
    return out


def _attempt(f, t, y, c, k1, h, order, rtol, atol):
    """One step: (y1, error norm, slopes)."""
    k = [k1]
    A, nodes = (_A5, _C5) if order == 5 else (_A8, _C8)
    for row, node in zip(A if order == 5 else A[:-1], nodes):
        y1 = y + h * _sum(row, k)
        k.append(f(t + node * h, y1, c))
    if order == 5:
        sk = atol + rtol * torch.maximum(y.abs(), y1.abs())
        return y1, torch.sqrt(((h * _sum(_E5, k) / sk) ** 2).mean(0)), k
    bs = _sum(A[-1], k)
    y1 = y + h * bs
    sk = atol + rtol * torch.maximum(y.abs(), y1.abs())
    e5 = ((_sum(_E8, k) / sk) ** 2).sum(0)
    e3 = (((bs - sum(w * k[j] for j, w in _B3.items())) / sk) ** 2).sum(0)
    den = e5 + 0.01 * e3
    den = torch.where(den <= 0, torch.ones_like(den), den)
    return y1, h.abs() * e5 * torch.sqrt(1 / (y.shape[0] * den)), k


def _hinit(f, t, y, c, f0, hmax, order, rtol, atol):
    sk = atol + rtol * y.abs()
    dnf, dny = ((f0 / sk) ** 2).sum(0), ((y / sk) ** 2).sum(0)
    h = torch.where((dnf <= 1e-10) | (dny <= 1e-10), torch.full_like(dnf, 1e-6), torch.sqrt(dny / dnf) * 0.01)
    h = torch.minimum(h, hmax)
    der2 = torch.sqrt((((f(t + h, y + h * f0, c) - f0) / sk) ** 2).sum(0)) / h
    der = torch.maximum(der2, torch.sqrt(dnf))
    h1 = torch.where(der <= 1e-15, torch.clamp(h * 1e-3, min=1e-6), (0.01 / der) ** (1 / order))
    return torch.minimum(torch.minimum(100 * h, h1), hmax)


_CTL = {5: (0.04, 0.2 - 0.04 * 0.75, 5.0, 10.0), 8: (0.1, 1 / 8 - 0.1 * 0.2, 1 / 0.3, 6.0)}


def _interval(f, t, y, c, dt, order, rtol, atol, nsteps=500):
    """One integrate(t + dt) call per tracer, restarted with an automatic first step: (t, y, ok)."""
    beta, expo, shrink, grow = _CTL[order]
    n = t.numel()
    xend = t + dt
    hmax = (xend - t).abs()
    t, y = t.clone(), y.clone()
    k1 = f(t, y, c)
    h = _hinit(f, t, y, c, k1, hmax, order, rtol, atol)
    fold = torch.full_like(t, 1e-4)
    rej = torch.zeros(n, dtype=torch.bool, device=t.device)
    ok = torch.ones_like(rej)
    idx = torch.arange(n, device=t.device)
    for it in range(nsteps + 1):
        if idx.numel() == 0:
            break
        ti, yi, hi, ci, xi, fo, rj = t[idx], y[:, idx], h[idx], c[:, idx], xend[idx], fold[idx], rej[idx]
        last = ti + 1.01 * hi - xi > 0
        hi = torch.where(last, xi - ti, hi)
        y1, err, k = _attempt(f, ti, yi, ci, k1[:, idx], hi, order, rtol, atol)
        acc = err <= 1
        fac11 = err ** expo
        hnew = hi / torch.clamp(fac11 / fo ** beta / 0.9, 1 / grow, shrink)
        hacc = torch.minimum(hnew, hmax[idx])
        hacc = torch.where(rj, torch.minimum(hacc, hi), hacc)
        hrej = hi / (shrink if order == 8 else torch.clamp(fac11 / 0.9, max=shrink))
        h[idx] = torch.where(acc, torch.where(last, hnew, hacc), hrej)
        rej[idx] = torch.where(acc, rj & last, torch.ones_like(acc))
        fold[idx] = torch.where(acc, torch.clamp(err, min=1e-4), fo)
        t[idx] = torch.where(acc, ti + hi, ti)
        y[:, idx] = torch.where(acc, y1, yi)
        k1[:, idx] = torch.where(acc, k[-1] if order == 5 else f(ti + hi, y1, ci), k1[:, idx])
        idx = idx[~(acc & last)]
    ok[idx] = False
    return t, y, ok


def _rowbuf(n, rows):
    return torch.zeros((n, rows, 7), dtype=torch.float64, device=_dev())


def _put(rows, nrows, j, t, values):
    """One more row of tracers j (columns of values), where there is room."""
    at = torch.clamp(nrows[j].long(), max=rows.shape[1] - 1)
    rows[j, at, 0] = t
    rows[j, at, 1:1 + values.shape[0]] = values.T
    nrows[j] += 1


def _answer(y, t, mode, status, rows, nrows, want, mu=None):
    n = t.numel()
    full = torch.zeros((6, n), dtype=torch.float64, device=t.device)
    full[:y.shape[0]] = y
    out = {"pos": full[:3], "mom": full[3:], "t": t, "mode": mode, "status": status}
    if mu is not None:
        out["mu"] = mu
    if want:
        out["rows"], out["nrows"] = rows, nrows
    return out


def _advance(f, order, t, y, c, dt, stop, rtol, atol, maxrows, ahead=False):
    """advance() of one mode: rows every dt until t reaches stop. Returns (row time, y, status, rows, nrows)."""
    n = t.numel()
    rows, nrows = _rowbuf(n, maxrows), torch.zeros(n, dtype=torch.int32, device=t.device)
    status = torch.zeros_like(nrows)
    trow = t.clone()
    t, y = t.clone(), y.clone()
    idx = torch.nonzero(t < stop)[:, 0]
    while idx.numel():
        rowt = t[idx] + dt[idx]
        ti, yi, ok = _interval(f, t[idx], y[:, idx], c[:, idx], dt[idx], order, rtol, atol)
        t[idx], y[:, idx] = ti, yi
        trow[idx] = rowt if ahead else ti
        _put(rows, nrows, idx, trow[idx], yi)
        status[idx[~ok]] = 2
        idx = idx[ok & (ti < stop[idx])]
    return trow, y, status, rows, nrows


def _dense(f, t, y, c, dt, stop, rtol, atol, maxrows):
    """Guiding centres with dense output: one integration through the call, rows from the continuous extension."""
    n = t.numel()
    beta, expo, shrink, grow = _CTL[5]
    rows, nrows = _rowbuf(n, maxrows), torch.zeros(n, dtype=torch.int32, device=t.device)
    trow, t, y, yrow = t.clone(), t.clone(), y.clone(), y.clone()
    k1 = f(t, y, c)
    hmax = 16 * dt
    h = _hinit(f, t, y, c, k1, hmax, 5, rtol, atol)
    fold, rej = torch.full_like(t, 1e-4), torch.zeros(n, dtype=torch.bool, device=t.device)
    idx = torch.arange(n, device=t.device)
    while idx.numel():
        ti, yi, hi, ci, fo, rj = t[idx], y[:, idx], h[idx], c[:, idx], fold[idx], rej[idx]
        y1, err, k = _attempt(f, ti, yi, ci, k1[:, idx], hi, 5, rtol, atol)
        acc = err <= 1
        fac11 = err ** expo
        hacc = torch.minimum(hi / torch.clamp(fac11 / fo ** beta / 0.9, 1 / grow, shrink), hmax[idx])
        hacc = torch.where(rj, torch.minimum(hacc, hi), hacc)
        h[idx] = torch.where(acc, hacc, hi / torch.clamp(fac11 / 0.9, max=shrink))
        rej[idx] = ~acc
        fold[idx] = torch.where(acc, torch.clamp(err, min=1e-4), fo)
        tn = torch.where(acc, ti + hi, ti)
        diff = y1 - yi
        bspl = hi * k[0] - diff
        r4, r5 = diff - hi * k[-1] - bspl, hi * _sum(_D5, k)
        for _ in range(17):
            tr = trow[idx] + dt[idx]
            due = acc & (tr <= tn) & (trow[idx] < stop[idx])
            if not bool(due.any()):
                break
            th = (tr - ti) / hi
            yr = yi + th * (diff + (1 - th) * (bspl + th * (r4 + (1 - th) * r5)))
            d, j = due, idx[due]
            trow[j], yrow[:, j] = tr[d], yr[:, d]
            _put(rows, nrows, j, tr[d], yr[:, d])
        t[idx], y[:, idx] = tn, torch.where(acc, y1, yi)
        k1[:, idx] = torch.where(acc, k[-1], k1[:, idx])
        idx = idx[trow[idx] < stop[idx]]
    return trow, yrow, torch.zeros_like(nrows), rows, nrows


# ---- the adaptive switch
def _cycper(m, t, X, gamma, mass, q):
    return 2 * np.pi * gamma * mass / _unit(m, t, X)[1] / q.abs()


def _lengthscale(m, t, X):
    Bs = _around(m, t, X)
    J = torch.stack([((Bs[:, 1 + 2 * a] - Bs[:, 2 + 2 * a]) / (2 * m.gradstep)).abs().amax(0) for a in range(3)])
    return torch.sqrt((Bs[:, 0] ** 2).sum(0)) / J.amax(0)


def _slow(m, t, X, cycper, eps=5e-2):
    """The time criterion: cyclotron period against |B| / |d|B|/dt|."""
    dB = (_unit(m, t + m.timestep, X)[1] - _unit(m, t - m.timestep, X)[1]) / m.timestep / 2
    return cycper * dB.abs() / _unit(m, t, X)[1] < eps


def _particle_adiabatic(m, t, y, mass, q, eps=5e-2):
    X, p = y[:3], y[3:]
    gm = torch.sqrt(mass ** 2 + (p * p).sum(0) / C ** 2)
    v = p / gm
    gamma = gm / mass
    b, mag = _unit(m, t, X)
    vpar = (v * b).sum(0)
    vperp = torch.sqrt((v * v).sum(0) - vpar ** 2)
    ok = gamma * mass * vperp / (q.abs() * mag) / _lengthscale(m, t, X) < eps
    return ok if m.static else ok & _slow(m, t, X, _cycper(m, t, X, gamma, mass, q))


def _gc_speed(pp, mass, mu, mag, par2):
    gamma = torch.sqrt(1 + 2 * mu * mag / (mass * C * C) + par2)
    slow = gamma - 1 < 1e-6
    v = torch.where(slow, torch.sqrt(2 * mu * mag / mass + (pp / mass) ** 2), C * torch.sqrt(1 - 1 / gamma ** 2))
    return v, torch.where(slow, pp / mass, pp / mass / gamma)


def _gc_adiabatic(m, t, y, mu, mass, q, eps=5e-2):
    X, pp = y[:3], y[3]
    mag = _unit(m, t, X)[1]
    v, vp = _gc_speed(pp, mass, mu, mag, (pp / mass / C) ** 2)
    g = 1 / torch.sqrt(1 - (v / C) ** 2)
    ok = g * mass * torch.sqrt((v - vp) * (v + vp)) / (q.abs() * mag) / _lengthscale(m, t, X) < eps
    if m.static:
        return ok
    v2, _ = _gc_speed(pp, mass, mu, mag, pp ** 2)  # the reference's gamma here takes ppar^2 in SI units
    return ok & _slow(m, t, X, _cycper(m, t, X, 1 / torch.sqrt(1 - (v2 / C) ** 2), mass, q))


def _to_gc(m, t, y, mass, q):
    """Guiding centre by fixed point R = r - rho(R): (x, y, z, ppar), mu."""
    r, p = y[:3], y[3:]
    gm = torch.sqrt(mass ** 2 + (p * p).sum(0) / C ** 2)
    v, gamma = p / gm, gm / mass

    def gyro(X):
        B = m.B(t, X)
        return gamma * mass / (q * (B * B).sum(0)) * _cross(B, v)

    R = r - gyro(r)
    open_ = torch.ones_like(mass, dtype=torch.bool)
    for _ in range(20):
        new = r - gyro(R)
        off = torch.sqrt(((new - R) ** 2).sum(0)) / torch.sqrt((new ** 2).sum(0))
        R = torch.where(open_, new, R)
        open_ = open_ & ~(off < 1e-3)
        if not bool(open_.any()):
            break
    b, mag = _unit(m, t, R)
    vp, sp = (v * b).sum(0), torch.sqrt((v * v).sum(0))
    out = torch.zeros_like(y)
    out[:3], out[3] = R, mass * gamma * vp
    return out, gamma ** 2 * mass * (sp - vp) * (sp + vp) / (2 * mag)


def _to_particle(m, t, y, mu, mass, q):
    """A particle on the gyro-circle at gyrophase 0 (its field taken at t = 0, as the reference does)."""
    X, pp = y[:3], y[3]
    mag = _unit(m, t, X)[1]
    g2 = 1 + 2 * mu * mag / (mass * C * C) + (pp / mass / C) ** 2
    v = torch.where(torch.sqrt(g2) - 1 < 1e-6, torch.sqrt(2 * mu * mag / mass + (pp / mass) ** 2),
                    C * torch.sqrt(1 - 1 / g2))
    vpar = pp / mass / torch.sqrt(g2)
    b, bn = _unit(m, torch.zeros_like(t), X)
    pa, gamma = torch.acos(vpar / v), 1 / torch.sqrt(1 - (v / C) ** 2)
    rc = gamma * mass * torch.sqrt((v - vpar) * (v + vpar)) / (q.abs() * bn)
    one, zero = torch.ones_like(bn), torch.zeros_like(bn)
    u = torch.stack([one, one, -(b[0] + b[1]) / b[2]])
    for a in (2, 1, 0):  # a vanishing component gives that axis, x before y before z
        axis = torch.stack([one if k == a else zero for k in range(3)])
        u = torch.where(b[a] == 0, axis, u)
    u = u / torch.sqrt((u * u).sum(0))
    vel = v * (torch.cos(pa) * b - torch.sign(q) * torch.sin(pa) * _cross(b, u))
    gv = 1 / torch.sqrt(1 - (vel * vel).sum(0) / C ** 2)
    return torch.cat([X + rc * u, mass * gv * vel])


def _adaptive(m, y, mass, q, delta, gcdt, cycres, rtol, atol, maxrows):
    n = mass.numel()
    dev = mass.device
    t = torch.zeros(n, dtype=torch.float64, device=dev)
    tcur, trow, stop, dt, gm, mu = (torch.zeros_like(t) for _ in range(6))
    mode = torch.zeros(n, dtype=torch.int8, device=dev)
    new, done = torch.ones(n, dtype=torch.bool, device=dev), torch.zeros(n, dtype=torch.bool, device=dev)
    seg = torch.zeros(n, dtype=torch.int32, device=dev)
    rows, nrows = _rowbuf(n, maxrows), torch.zeros(n, dtype=torch.int32, device=dev)
    status = torch.zeros_like(nrows)
    rhs = (_particle_rhs(m), _gc_rhs(m))

    def gc_at_start(j):
        ok = _particle_adiabatic(m, trow[j], y[:, j], mass[j], q[j])
        j = j[ok]
        y[:, j], mu[j] = _to_gc(m, trow[j], y[:, j], mass[j], q[j])
        mode[j] = 1

    def begin(j, left):
        if not j.numel():
            return
        t[j] = trow[j]
        stop[j] = trow[j] + left
        p = y[3:, j]
        gm[j] = torch.sqrt(mass[j] ** 2 + (p * p).sum(0) / C ** 2)
        per = _cycper(m, trow[j], y[:3, j], gm[j] / mass[j], mass[j], q[j]) / cycres
        dt[j] = torch.where(mode[j] == 1, torch.full_like(per, gcdt), per)
        new[j] = False

    def put(j, values):
        _put(rows, nrows, j, trow[j], values)

    gc_at_start(torch.arange(n, device=dev))
    while not bool(done.all()):
        j = torch.nonzero(new & ~done)[:, 0]
        begin(j, torch.where(seg[j] > 0, delta[j] - tcur[j], delta[j]))
        over = ~done & ~(t < stop)
        done |= over & ~(tcur < delta)
        j = torch.nonzero(over & ~done)[:, 0]  # time left within the advance: another segment
        seg[j] += 1
        begin(j, delta[j] - tcur[j])
        for md in (0, 1):
            j = torch.nonzero(~done & ~new & (mode == md))[:, 0]
            if not j.numel():
                continue
            rowt = t[j] + dt[j]
            if md == 0:
                ti, yi, ok = _interval(rhs[0], t[j], y[:, j], torch.stack([q[j], mass[j], gm[j]]), dt[j], 8, rtol, atol)
                t[j], y[:, j], trow[j], tcur[j] = ti, yi, rowt, ti + dt[j]
                put(j, yi)
                go = ok & _particle_adiabatic(m, rowt, yi, mass[j], q[j])
            else:
                ti, yi, ok = _interval(rhs[1], t[j], y[:4, j], torch.stack([q[j], mu[j], mass[j]]), dt[j], 5, rtol, atol)
                y[:4, j] = yi
                t[j], trow[j], tcur[j] = ti, ti, ti
                put(j, yi)
                go = ok & ~_gc_adiabatic(m, ti, yi, mu[j], mass[j], q[j])
            status[j[~ok]] = 2
            done[j[~ok]] = True
            j = j[go]
            if not j.numel():
                continue
            if md == 0:
                g, mu[j] = _to_gc(m, trow[j], y[:, j], mass[j], q[j])
                y[:, j] = g
                sp = g[:4].clone()
                p2 = (yi[3:, go] ** 2).sum(0)
                put(j, torch.cat([sp, mu[j][None], (torch.sqrt(p2) / torch.sqrt(mass[j] ** 2 + p2 / C ** 2))[None]]))
            else:
                y[:, j] = _to_particle(m, trow[j], y[:4, j], mu[j], mass[j], q[j])
                put(j, y[:, j])
            mode[j] = 1 - md
            t[j] = tcur[j] = trow[j]
            seg[j] += 1
            new[j] = True
    y[4:, mode == 1] = 0
    return trow, y, mode, mu, status, rows, nrows


# ---- field lines
_RKF_B = [[], [.25], [.09375, .28125], [8.793809740555303e-1, -3.277196176604461, 3.320892125625853],
          [2.032407407407407, -8.0, 7.173489278752436, -2.058966861598441e-1],
          [-2.962962962962963e-1, 2.0, -1.381676413255361, 4.529727095516569e-1, -.275]]
_RKF_R = [2.777777777777778e-3, 0, -2.994152046783626e-2, -2.919989367357789e-2, .02, 3.636363636363636e-2]
_RKF_C = [1.157407407407407e-1, 0, 5.489278752436647e-1, 5.353313840155945e-1, -.2, 0]


def _mag(m, X):
    return _unit(m, torch.zeros_like(X[0]), X)[1]


def _trace(m, X, Bm, resolution=50.0, cap=1024):
    """s and |B| along the field lines through X out to |B| > Bm both ways, RKF45 steps of at most a fiftieth of the
    curvature radius: (s, B, first, count), the start in column cap."""
    n = X.shape[1]
    dev = X.device
    B = _unit(m, torch.zeros(n, device=dev, dtype=torch.float64), X)
    Bv, mag, d = B[0] * B[1], B[1], m.gradstep
    g = torch.stack([(_mag(m, _shift(X, a, d)) - _mag(m, _shift(X, a, -d))) / (2 * d) for a in range(3)])
    gp = g - g * mag / mag ** 2 * Bv
    ds = mag / torch.sqrt((gp * gp).sum(0)) / resolution
    S = torch.zeros((n, 2 * cap), dtype=torch.float64, device=dev)
    Bs = torch.full_like(S, float("inf"))
    Bs[:, cap] = mag
    # both directions of every line together: line k and, backward, line k + n
    one = torch.ones(n, dtype=torch.float64, device=dev)
    sign, tol, step = torch.cat([one, -one]), torch.cat([1e-3 * one, 1e-4 * one]), torch.cat([ds, ds])
    x = torch.cat([torch.zeros((1, 2 * n), dtype=torch.float64, device=dev), torch.cat([X, X], dim=1)])
    pos = torch.full((2 * n,), cap, dtype=torch.long, device=dev)
    t, h = torch.zeros_like(step), step.clone()
    idx = torch.arange(2 * n, device=dev)
    while idx.numel():
        top, sg = step[idx], sign[idx]
        hi = torch.where(t[idx] + h[idx] > top, top - t[idx], h[idx])
        k = []
        for row in _RKF_B:
            xt = x[:, idx] + (_sum(row, k) if row else 0.0)
            k.append(hi * sg * torch.cat([torch.ones_like(hi)[None], _unit(m, torch.zeros_like(hi), xt[1:])[0]]))
        r = (_sum(_RKF_R, k).abs() / hi).amax(0)
        acc = r <= tol[idx]
        x[:, idx] = torch.where(acc, x[:, idx] + _sum(_RKF_C, k), x[:, idx])
        t[idx] = torch.where(acc, t[idx] + hi, t[idx])
        j = idx[acc]
        pos[j] += sign[j].long()
        S[j % n, pos[j]] = x[0, j]
        Bs[j % n, pos[j]] = _mag(m, x[1:, j])
        h[idx] = torch.minimum(hi * torch.clamp(0.84 * (tol[idx] / r) ** 0.25, 0.1, 4.0), top)
        full = ~(t[idx] < top)
        end = full & (Bs[idx % n, pos[idx]] > Bm[idx % n])
        t[idx] = torch.where(full, torch.zeros_like(hi), t[idx])
        h[idx] = torch.where(full, top, h[idx])
        idx = idx[~end & (pos[idx] > 1) & (pos[idx] < 2 * cap - 2)]
    return S, Bs, pos[n:], pos[:n] - pos[n:] + 1


def _line_integral(m, X, Bm, inverse):
    """Half-bounce path (integral of 1 / sqrt(1 - B/Bm), where `inverse`) or second invariant (sqrt(1 - B/Bm)) of every
    line on the quadratic interpolating spline of |B|(s) (knots midway between the inner points), mirror point to
    mirror point."""
    S, Bs, first, count = _trace(m, X, Bm)
    n, dev = X.shape[1], X.device
    col = torch.arange(S.shape[1], device=dev)
    on = (col >= first[:, None]) & (col < (first + count)[:, None])
    inside = on & torch.where(inverse[:, None], Bs <= Bm[:, None], Bs < Bm[:, None])
    fin = torch.where(inside.any(1), inside.int().argmax(1), first)
    lin = torch.where(inside.any(1), S.shape[1] - 1 - inside.int().flip(1).argmax(1), first)
    lo = torch.maximum(fin - 1, first)
    cnt = torch.minimum(lin + 1, first + count - 1) - lo + 1
    top = int(cnt.max())
    at = torch.clamp(lo[:, None] + torch.arange(top, device=dev), max=S.shape[1] - 1)
    s, b = S.gather(1, at), Bs.gather(1, at)
    live = torch.arange(top, device=dev)[None, :] < cnt[:, None]
    lastc = (cnt - 1)[:, None]
    s = torch.where(live, s, s.gather(1, lastc))
    b = torch.where(live, b, b.gather(1, lastc))
    # knots T[j], j = 0 .. cnt + 2
    j = torch.arange(top + 3, device=dev)[None, :]
    mid = (s.gather(1, torch.clamp(j - 2, 0, top - 1).expand(n, -1)) + s.gather(1, torch.clamp(j - 1, 0, top - 1).expand(n, -1))) / 2
    T = torch.where(j <= 2, s[:, :1], torch.where(j >= cnt[:, None], s.gather(1, lastc), mid))

    def basis(v, l):
        """The three B-splines alive on knot panel l at v, for v and l of one shape [n, k]."""
        T0, T1, T2, T3 = (T.gather(1, torch.clamp(l + o, 0, top + 2)) for o in (-1, 0, 1, 2))
        w1 = (T2 - v) / (T2 - T1)
        w2 = 1 - w1
        a = (T2 - v) / (T2 - T0)
        c = (v - T1) / (T3 - T1)
        return w1 * a, w1 * (1 - a) + w2 * (1 - c), w2 * c

    # collocation rows: point i lies on panel clamp(i + 1, 2, cnt - 1); tridiagonal
    i = torch.arange(top, device=dev)[None, :].expand(n, -1)
    l = torch.minimum(torch.clamp(i + 1, min=2), lastc)
    h = basis(s, l)
    low, dia, upp = torch.zeros_like(s), torch.zeros_like(s), torch.zeros_like(s)
    for o in range(3):
        w, k = h[o], l + o - 2
        low = torch.where(k == i - 1, w, low)
        dia = torch.where(k == i, w, dia)
        upp = torch.where(k == i + 1, w, upp)
    dia = torch.where(live, dia, torch.ones_like(dia))
    low, upp = torch.where(live, low, torch.zeros_like(low)), torch.where(live, upp, torch.zeros_like(upp))
    cf, dd = b.clone(), dia.clone()
    for k in range(1, top):
        w = low[:, k] / dd[:, k - 1]
        dd[:, k] = dd[:, k] - w * upp[:, k - 1]
        cf[:, k] = cf[:, k] - w * cf[:, k - 1]
    cf[:, -1] = cf[:, -1] / dd[:, -1]
    for k in range(top - 2, -1, -1):
        cf[:, k] = (cf[:, k] - upp[:, k] * cf[:, k + 1]) / dd[:, k]

    def spline(v, l):
        w = basis(v, l)
        return sum(w[o] * cf.gather(1, torch.clamp(l + o - 2, 0, top - 1)) for o in range(3))

    def mirror(a, c, l):
        """The mirror point between the outermost two points, by bisection."""
        a, c, l = a[:, None].clone(), c[:, None].clone(), l[:, None]
        up = spline(c, l) > Bm[:, None]
        for _ in range(80):
            v = (a + c) / 2
            hi = (spline(v, l) > Bm[:, None]) == up
            a, c = torch.where(hi, a, v), torch.where(hi, v, c)
        return ((a + c) / 2)[:, 0]

    two = torch.full_like(lo, 2)
    sa = mirror(s[:, 0], s[:, 1], two)
    sb = mirror(s.gather(1, torch.clamp(lastc - 1, min=0))[:, 0], s.gather(1, lastc)[:, 0], torch.clamp(cnt - 1, min=2))
    mid, half = (sa + sb) / 2, (sb - sa) / 2
    gx, gw = (_T(a) for a in np.polynomial.legendre.leggauss(16))
    ang = torch.asin(torch.clamp((T - mid[:, None]) / half[:, None], -1, 1))
    total = torch.zeros(n, dtype=torch.float64, device=dev)
    per = max(1, (1 << 25) // (16 * n))  # panels at once
    for p0 in range(2, top, per):
        p = torch.arange(p0, min(p0 + per, top), device=dev)
        ea, eb = ang[:, p], ang[:, p + 1]
        th = (((ea + eb) / 2)[..., None] + ((eb - ea) / 2)[..., None] * gx).reshape(n, -1)
        panel = p.repeat_interleave(16)[None, :].expand(n, -1)
        arg = 1 - spline(mid[:, None] + half[:, None] * torch.sin(th), panel) / Bm[:, None]
        root = torch.sqrt(torch.clamp(arg, min=0))
        val = torch.where(inverse[:, None], torch.where(arg > 0, 1 / root, torch.zeros_like(root)), root)
        part = (eb - ea) / 2 * ((val * half[:, None] * torch.cos(th)).reshape(n, -1, 16) * gw).sum(-1)
        total = total + torch.where((p < cnt[:, None]) & (eb > ea), part, torch.zeros_like(part)).sum(1)
    # three points of a half-bounce path: the equatorial bounce
    s12, s23, s13 = s[:, 0] - s[:, 1], s[:, 1] - s[:, 2], s[:, 0] - s[:, 2]
    B2 = 2 * (b[:, 0] * s23 - b[:, 1] * s13 + b[:, 2] * s12) / (s12 * s13 * s23)
    total = torch.where(inverse & (cnt == 3), np.pi * torch.sqrt(2 * Bm / B2), total)
    # a line that stays above the mirror field has no second invariant
    low_b = torch.where(on, Bs, torch.full_like(Bs, float("inf"))).amin(1)
    return torch.where(~inverse & ((low_b > Bm) | ((low_b - Bm).abs() / Bm < 1e-12)), torch.zeros_like(total), total)


def _half_bounce(m, X, Bm):
    return _line_integral(m, X, Bm, torch.ones_like(Bm, dtype=torch.bool))


def _bounce_period(m, y, mu, mass):
    mag, pp = _mag(m, y[:3]), y[3]
    gamma = torch.sqrt(1 + 2 * mu * mag / (mass * C * C) + (pp / (mass * C)) ** 2)
    slow = gamma - 1 < 1e-6
    p = torch.where(slow, torch.sqrt(2 * mass * mu * mag + pp ** 2), mass * C * torch.sqrt((gamma + 1) * (gamma - 1)))
    v = torch.where(slow, p / mass, p / mass / gamma)
    Bm = torch.where(slow, p * p / (2 * mass * mu), p * p / ((p - pp) * (p + pp)) * mag)
    return 2 / v * _half_bounce(m, y[:3], Bm)


def _bc_rhs(m, d):
    def f(t, y, c):
        Bm, kdrift = c[0], c[1]
        B = m.B(t, y)
        b = B / torch.sqrt((B * B).sum(0))
        r = torch.stack([y[0], y[1], torch.zeros_like(y[0])]) / torch.maximum(y[0].abs(), y[1].abs())
        r = r - (r * b).sum(0) * b
        r = r / torch.sqrt((r * r).sum(0))
        w = _cross(b, r)
        lines = torch.cat([y + d * r, y - d * r, y + d * w, y - d * w, y, y], dim=1)
        path = torch.arange(6, device=Bm.device).repeat_interleave(Bm.numel()) == 5
        I = _line_integral(m, lines, Bm.repeat(6), path).reshape(6, -1)

        def diff(up, um):  # one-sided where the line at one end lies above the mirror field
            central = torch.where(um == 0, (up - I[4]) / d, (up - um) / (2 * d))
            return torch.where(up == 0, (I[4] - um) / d, central)

        g = diff(I[0], I[1]) * r + diff(I[2], I[3]) * w
        return kdrift / (I[5] * (B * B).sum(0)) * _cross(g, B)
    return f


def _exact_bc(case, w):
    n, p = case["n"], w["params"]
    m = _Double()
    pos, v, mass, q = _T(w["pos"].T), _T(w["v"]), _T(w["mass"]), _T(w["charge"])
    gamma = 1 / torch.sqrt(1 - (v / C) ** 2)
    mu = (gamma * v * torch.sin(torch.deg2rad(_T(w["eqpa"])))) ** 2 * mass / (2 * _mag(m, pos))
    Bm = mass * gamma ** 2 * v ** 2 / (2 * mu)
    dt = p["bctimestep"] * 2 / v * _half_bounce(m, pos, Bm)
    K = torch.ceil(case["delta"] / dt)
    c = torch.stack([Bm, gamma * mass * v * v / q])
    f = _bc_rhs(m, p["eyegradientstep"])
    rows = torch.zeros((n, 16, 4), dtype=torch.float64, device=pos.device)
    t, y = torch.zeros(n, dtype=torch.float64, device=pos.device), pos.clone()
    for j in range(int(K.max())):
        i = torch.nonzero(K > j)[:, 0]
        _, y[:, i], _ = _interval(f, t[i], y[:, i], c[:, i], dt[i], 5, p["rtol"], p["atol"])
        t[i] = j * dt[i]
        if j < 16:
            rows[i, j, 0], rows[i, j, 1:] = t[i], y[:, i].T
    return {"state": torch.cat([t[None], y, t[None]]).T.contiguous(), "rows": rows, "nrows": K.to(torch.int32),
            "status": torch.zeros(n, dtype=torch.int32)}


def exact(case, seed):
    w, kind, delta = _workload(case, seed)
    if kind == "bc":
        return _exact_bc(case, w)
    n, p, fam = case["n"], w["params"], case["family"]
    want = _wants_rows(case)
    mass, q = _T(w["mass"]), _T(w["charge"])
    dur = _T(np.broadcast_to(np.asarray(delta, float), (n,)))
    t0 = torch.full((n,), 0.5 if fam == "grid" else 0.0, dtype=torch.float64, device=mass.device)
    rtol, atol, rows = p["rtol"], p["atol"], _max_rows(case) if want else 1
    if kind == "gc":
        m = _Gridded(_dipole_grid(case["nodes"])) if fam == "grid" else _Double()
        pos, v = _T(w["pos"].T), _T(w["v"])
        gamma = 1 / torch.sqrt(1 - (v / C) ** 2)
        vpar = v * torch.cos(_T(w["pa"]) * (np.pi / 180))
        mu = gamma ** 2 * mass * (v - vpar) * (v + vpar) / (2 * _unit(m, t0, pos)[1])
        y, c = torch.cat([pos, (gamma * mass * vpar)[None]]), torch.stack([q, mu, mass])
        dt = torch.full_like(mass, p["gctimestep"])
        if fam == "bounce":
            dt = _bounce_period(m, y, mu, mass) / case["resolution"]
        step = _dense if p.get("dense_output") else lambda f, *a: _advance(f, 5, *a)
        t, y, status, rw, nr = step(_gc_rhs(m), t0, y, c, dt, t0 + dur, rtol, atol, rows)
        return _answer(y, t, torch.ones(n, dtype=torch.int8), status, rw, nr, want)
    vel = _T(w["vel"].T)
    gamma = 1 / torch.sqrt(1 - (vel * vel).sum(0) / C ** 2)
    y = torch.cat([_T(w["pos"].T), mass * gamma * vel])
    if kind == "adaptive":
        m = _Harris() if case["field"] == "Harris" else _Breathing()
        t, y, mode, mu, status, rw, nr = _adaptive(m, y, mass, q, dur, p["gctimestep"], 10.0, rtol, atol, rows)
        return _answer(y, t, mode, status, rw, nr, want, mu)
    m = _Earth()
    gm = torch.sqrt(mass ** 2 + (y[3:] ** 2).sum(0) / C ** 2)
    dt = _cycper(m, t0, y[:3], gm / mass, mass, q) / case["resolution"]
    t, y, status, rw, nr = _advance(_particle_rhs(m), 8, t0, y, torch.stack([q, mass, gm]), dt, t0 + dur, rtol, atol,
                                    rows, ahead=True)
    return _answer(y, t, torch.zeros(n, dtype=torch.int8), status, rw, nr, want)
