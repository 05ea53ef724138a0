"""Guiding centres and particles worked on by teams of lanes (small ensembles, the
end of a launch) end in the same bits as one tracer a lane: a tracer's result
does not depend on how many others are advanced with it."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu

BIG = 20011  # more than three rounds of four-tracer warps: one tracer a lane until the end of the launch


def _grid_field():
    return W.dipole_grid(41, 41, 21)


def _static_grid_field():
    g = W.dipole_grid(41, 41, 21)
    g.static = True
    return g


MODELS = {"EarthDipole": F.EarthDipole, "DoubleDipole": F.DoubleDipole, "VarEarthDipole": F.VarEarthDipole,
          "CompressedDipole": F.CompressedDipole, "Harris": F.Harris, "UniformCrossedEB": lambda: F.UniformCrossedEB(1e-4, 1e-7),
          "Grid": _grid_field, "StaticGrid": _static_grid_field}


def _run(field, kind, n, w, delta, **cfg):
    from rapt_gb300 import Ensemble
    ens = Ensemble(field, n, max_rows=48, max_switch=8)
    ens.configure(rtol=1e-7, atol=1e-7, **cfg)
    if kind == "gc":
        ens.set_guiding_centers(w["pos"][:n], w["v"][:n], pa=w["pa"][:n], t0=0.5, mass=w["mass"][:n], charge=w["charge"][:n])
    else:
        ens.set_particles(w["pos"][:n], w["vel"][:n], 0.5, w["mass"][:n], w["charge"][:n])
    ens.upload()
    if kind == "adaptive":
        ens.adaptive_init()
    ens.advance(kind, delta)
    h = ens.download()
    rows, mode, nrows, _, _ = ens.rows()
    k = min(n, 128)
    return [h[a][..., :k].copy() for a in ("s", "t_row", "mu", "status", "mode", "naccept", "nreject", "nfcn")] + \
        [nrows[:k].copy(), [rows[i, :nrows[i]].copy() for i in range(k)]]


def _same(a, b, n):
    for x, y in zip(a[:-1], b[:-1]):
        assert np.array_equal(x[..., :n], y[..., :n], equal_nan=x.dtype.kind == "f")
    for x, y in zip(a[-1][:n], b[-1][:n]):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("eom", [0, 1, 2])
def test_guiding_centre_teams(model, eom):
    field = MODELS[model]()
    w = W.config2(BIG, seed=5)
    if model in ("Harris", "UniformCrossedEB"):
        w = dict(w, mass=np.full(BIG, W.m_pr), charge=np.full(BIG, W.e), v=np.linspace(3e5, 3e6, BIG),
                 pos=W.config3(BIG, 2)["pos"])
    delta = 0.02 if model in ("Grid", "StaticGrid") else 0.05
    cfg = dict(gctimestep=0.01, gc_eom=eom)
    big = _run(field, "gc", BIG, w, delta, **cfg)
    for n in (1, 7, 128):
        _same(_run(field, "gc", n, w, delta, **cfg), big, n)


@pytest.mark.parametrize("model", ["DoubleDipole", "CompressedDipole"])
def test_dense_output_teams(model):
    w = W.config2(BIG, seed=6)
    cfg = dict(gctimestep=0.01, dense_output=1)
    big = _run(MODELS[model](), "gc", BIG, w, 0.1, **cfg)
    for n in (1, 33, 128):
        _same(_run(MODELS[model](), "gc", n, w, 0.1, **cfg), big, n)


@pytest.mark.parametrize("n", [1, 33, 2500])
@pytest.mark.parametrize("cfg", [{}, {"max_steps_per_launch": 7}, {"use_graph": 1}, {"blocks_per_sm": 1, "threads_per_block": 64}])
def test_adaptive_hand_over(n, cfg):
    """Adaptive in one launch (switched tracers handed over on the device) against
    one launch sequence per tracer: states, rows, switch logs and counters, with
    step budgets that end launches in mid-flight, graph replay and other grids."""
    from rapt_gb300 import Ensemble
    w = W.config3(4096, seed=11)
    d = 1.0 + 11.0 * np.random.default_rng(1).random(4096)
    out = []
    k = min(n, 64)
    for m, extra in ((n, cfg), (k, {"per_tracer_launches": 1})):
        ens = Ensemble(F.Harris(), m, max_rows=256, max_switch=16)
        ens.configure(rtol=1e-8, atol=1e-8, gctimestep=0.5, **extra)
        ens.set_particles(w["pos"][:m], w["vel"][:m], 0.0, w["mass"][:m], w["charge"][:m])
        ens.upload()
        ens.adaptive_init()
        ens.advance("adaptive", d[:m])
        h = ens.download()
        rows, mode, nrows, swt, swm = ens.rows()
        nsw = np.minimum(h["nswitch"][:k], 16)
        out.append([h[a][..., :k].copy() for a in ("s", "t_row", "tcur", "mu", "status", "mode", "naccept", "nfcn", "nswitch")] +
                   [nrows[:k].copy()] + [rows[i, :nrows[i]].copy() for i in range(k)] +
                   [mode[i, :nrows[i]].copy() for i in range(k)] + [swt[i, :nsw[i]].copy() for i in range(k)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 33, 609, 5000])
@pytest.mark.parametrize("tableau", [0, 1])
def test_particles_spread(n, tableau):
    """Few particles a warp (small ensembles) against full warps."""
    from rapt_gb300 import Ensemble
    w = W.config1(BIG)
    out = []
    for m in (n, BIG):
        ens = Ensemble(F.EarthDipole(), m, max_rows=32)
        ens.configure(rtol=1e-8, atol=1e-8, cyclotronresolution=10, tableau=tableau)
        ens.set_particles(w["pos"][:m], w["vel"][:m], 0.0, w["mass"][:m], w["charge"][:m])
        ens.upload()
        ens.advance("particle", 0.02)
        h = ens.download()
        k = min(n, 128)
        out.append([h[a][..., :k].copy() for a in ("s", "t_row", "status", "naccept", "nreject", "nfcn")])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [7297, 10007, 19457])
@pytest.mark.parametrize("model", ["DoubleDipole", "CompressedDipole", "Harris", "Grid"])
@pytest.mark.parametrize("cadence,dense", [(0.01, 0), (0.07, 0), (0.0, 0), (0.01, 1), (0.0, 1)])
def test_shared_between_warps(model, n, cadence, dense):
    """Tracers given from warp to warp inside an interval against a launch in which
    each stays where it began (a step budget, here far away, switches sharing off):
    states, rows and counters, with several intervals and with one, and durations
    that leave many warps without a tracer."""
    if cadence == 0.0 and model not in ("DoubleDipole", "CompressedDipole"):
        pytest.skip("a bounce needs mirror points")
    from rapt_gb300 import Ensemble
    w = W.config2(n, seed=9)
    if model == "Harris":
        w = dict(w, mass=np.full(n, W.m_pr), charge=np.full(n, W.e), v=np.linspace(3e5, 3e6, n), pos=W.config3(n, 2)["pos"])
    delta = np.random.default_rng(4).choice([0.0, 0.01, 0.03, 0.06], n)
    out = []
    for budget, graph in ((0, 0), (0, 1), (1 << 40, 0)):
        ens = Ensemble(MODELS[model](), n, max_rows=64)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=cadence, bounceresolution=20.0, dense_output=dense,
                      max_steps_per_launch=budget, use_graph=graph)
        ens.set_guiding_centers(w["pos"], w["v"], pa=w["pa"], t0=0.5, mass=w["mass"], charge=w["charge"])
        ens.upload()
        st = ens.advance("gc", delta)
        h = ens.download()
        rows, _, nrows, _, _ = ens.rows()
        out.append([h[a].copy() for a in ("s", "t_row", "tcur", "mu", "status", "flags", "naccept", "nreject", "nfcn")] +
                   [nrows, np.where(np.arange(64)[None, :, None] < nrows[:, None, None], rows, 0.0),
                    np.array([st[a] for a in ("accepted", "rejected", "rhs_evals", "done", "failed")])])
    for a, g, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
        assert np.array_equal(g, b, equal_nan=a.dtype.kind == "f")


def test_shared_rows_full_and_resume():
    """A row buffer that fills up: the tracers stop and are resumed, shared or not."""
    from rapt_gb300 import Ensemble
    n = 9001
    w = W.config2(n, seed=12)
    delta = np.random.default_rng(5).choice([0.01, 0.03, 0.06], n)
    out = []
    for budget in (0, 1 << 40):
        ens = Ensemble(F.DoubleDipole(), n, max_rows=4)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.01, max_steps_per_launch=budget)
        ens.set_guiding_centers(w["pos"], w["v"], pa=w["pa"], t0=0.5, mass=w["mass"], charge=w["charge"])
        ens.upload()
        ens.advance("gc", delta)
        got = []
        for _ in range(4):
            rows, _, nrows, _, _ = ens.rows()
            got += [nrows, np.where(np.arange(4)[None, :, None] < nrows[:, None, None], rows, 0.0)]
            ens.advance_resume("gc")
        h = ens.download()
        out.append(got + [h[a].copy() for a in ("s", "t_row", "status", "flags", "naccept", "nreject", "nfcn")])
    assert (out[0][0] == 3).any() and out[0][2].any()  # a row and its possible switch row have to fit
    for a, b in zip(*out):
        assert np.array_equal(a, b)
