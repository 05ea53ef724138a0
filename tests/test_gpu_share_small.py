"""Sharing between warps in ensembles of fewer tracers than sub-partitions hold at once
(from where a round of teams a sub-partition no longer takes them all), in every field
model, against a launch in which each tracer stays in its warp (a step budget, here far
away, switches sharing off): states, rows and counters."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MODELS = {"EarthDipole": F.EarthDipole, "DoubleDipole": F.DoubleDipole, "VarEarthDipole": F.VarEarthDipole,
          "CompressedDipole": F.CompressedDipole, "Harris": F.Harris, "Parabolic": lambda: F.Parabolic(20e-9, 2e-9, 0.2),
          "UniformBz": lambda: F.UniformBz(1e-7), "UniformCrossedEB": lambda: F.UniformCrossedEB(1e-4, 1e-7),
          "Grid": lambda: W.dipole_grid(41, 41, 21)}


@pytest.mark.parametrize("n", [1217, 2433, 7296, 9001])
@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("dense", [0, 1])
def test_shared_between_warps(model, n, dense):
    from rapt_gb300 import Ensemble
    w = W.config2(n, seed=13)
    if model in ("Harris", "Parabolic", "UniformBz", "UniformCrossedEB"):
        w = dict(w, mass=np.full(n, W.m_pr), charge=np.full(n, W.e), v=np.linspace(3e5, 3e6, n), pos=W.config3(n, 2)["pos"])
    delta = np.random.default_rng(4).choice([0.0, 0.01, 0.03, 0.06], n)
    out = []
    for budget in (0, 1 << 40):
        ens = Ensemble(MODELS[model](), n, max_rows=32)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.01, dense_output=dense, max_steps_per_launch=budget)
        ens.set_guiding_centers(w["pos"], w["v"], pa=w["pa"], t0=0.5, mass=w["mass"], charge=w["charge"])
        ens.upload()
        st = ens.advance("gc", delta)
        h = ens.download()
        rows, _, nrows, _, _ = ens.rows()
        out.append([h[a].copy() for a in ("s", "t_row", "tcur", "mu", "status", "flags", "naccept", "nreject", "nfcn")] +
                   [nrows, np.where(np.arange(32)[None, :, None] < nrows[:, None, None], rows, 0.0),
                    np.array([st[a] for a in ("accepted", "rejected", "rhs_evals", "done", "failed")])])
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")


@pytest.mark.parametrize("model", ["Parabolic", "UniformBz", "VarEarthDipole"])
@pytest.mark.parametrize("eom", [0, 1, 2])
def test_teams(model, eom):
    """Few tracers, worked on by teams of lanes, against the same among many."""
    from rapt_gb300 import Ensemble
    big = 20011
    w = W.config2(big, seed=14)
    if model != "VarEarthDipole":
        w = dict(w, mass=np.full(big, W.m_pr), charge=np.full(big, W.e), v=np.linspace(3e5, 3e6, big), pos=W.config3(big, 2)["pos"])
    out = []
    for n in (big, 1, 7, 128):
        ens = Ensemble(MODELS[model](), n, max_rows=16)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.01, gc_eom=eom)
        ens.set_guiding_centers(w["pos"][:n], w["v"][:n], pa=w["pa"][:n], t0=0.5, mass=w["mass"][:n], charge=w["charge"][:n])
        ens.upload()
        ens.advance("gc", 0.05)
        h = ens.download()
        out.append([h[a][..., :128].copy() for a in ("s", "t_row", "mu", "status", "naccept", "nreject", "nfcn")])
    for n, few in zip((1, 7, 128), out[1:]):
        for a, b in zip(out[0], few):
            assert np.array_equal(a[..., :n], b[..., :n], equal_nan=a.dtype.kind == "f")
