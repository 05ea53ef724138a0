"""Adaptive ensembles in one launch: what the hand-over between the two modes has to
keep besides the states (test_gpu_teams.py)."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _sheet(which, max_rows=256, **cfg):
    from rapt_gb300 import Ensemble
    w = W.config3(4096, seed=11)
    n = len(which)
    ens = Ensemble(F.Harris(), n, max_rows=max_rows, max_switch=16)
    ens.configure(rtol=1e-8, atol=1e-8, gctimestep=0.5, **cfg)
    ens.set_particles(w["pos"][which], w["vel"][which], 0.0, w["mass"][which], w["charge"][which])
    ens.upload()
    ens.adaptive_init()
    return ens


@pytest.fixture(scope="module")
def switching():
    """Tracers of the sheet by the number of their switches, most first."""
    ens = _sheet(np.arange(256), per_tracer_launches=1)
    ens.advance("adaptive", 12.0)
    nsw = ens.download()["nswitch"].copy()
    order = np.argsort(-nsw, kind="stable")
    assert nsw[order[4]] > 0
    return order


@pytest.mark.parametrize("n", [1, 2, 5])
def test_each_tracer_is_advanced_once(n, switching):
    """The counts of a call over few tracers (rings of as many entries, polled by
    every idle warp) are those of one launch sequence per tracer, call after call."""
    which = switching[:n]
    h = None
    for rep in range(20):
        ens = _sheet(which) if rep else _sheet(which, per_tracer_launches=1)
        st = ens.advance("adaptive", 12.0)
        d = ens.download()
        if not rep:
            h = {a: d[a].copy() for a in ("s", "naccept", "nreject", "nfcn", "nswitch")}
            continue
        for a in h:
            assert np.array_equal(d[a], h[a]), a
        assert st["accepted"] == d["naccept"].sum() and st["switches"] == d["nswitch"].sum()
        assert st["done"] == n and st["failed"] == 0


@pytest.mark.parametrize("cfg", [{}, {"blocks_per_sm": 1, "threads_per_block": 32}])
def test_a_step_budget_bounds_a_launch(cfg):
    """Several times as many tracers as a launch has lanes, and a budget of 100 attempts
    a lane: a launch that leaves tracers to the next ends within some ms, without waits
    (warps that wait in vain give up after 2^18 polls of a microsecond, 262 ms)."""
    n = 60000 if cfg else 200000
    which = np.arange(n) % 4096
    st = _sheet(which, max_rows=256, max_steps_per_launch=100, **cfg).advance("adaptive", 20.0)
    assert st["done"] == n and st["failed"] == 0
    assert st["launches"] > 4 and st["kernel_ms"] < 60.0 * st["launches"], (st["kernel_ms"], st["launches"])


@pytest.mark.parametrize("n", [90000, 60000])
def test_one_mode_and_a_few_of_the_other(n):
    """Nearly all tracers in one mode (above 77,824 on 152 SMs most blocks are given to it)
    and a few that switch: states, counts and switches of one launch sequence per tracer."""
    from rapt_gb300 import Ensemble
    w = W.config4(n, 31)
    rng = np.random.default_rng(3)
    d = w["vel"] / np.linalg.norm(w["vel"], axis=1)[:, None]
    ke = 10 ** rng.uniform(4, 5, n)
    ke[:: n // 300] = 10 ** rng.uniform(6, 7, len(ke[:: n // 300]))  # protons that change between the modes
    mass = np.full(n, W.m_el)
    charge = np.full(n, -W.e)
    mass[:: n // 300] = W.m_pr
    charge[:: n // 300] = W.e
    vel = d * W.speed_from_ke(ke, mass)[:, None]
    out = []
    for idx in (np.arange(n), np.arange(n)[:: n // 300]):
        ens = Ensemble(F.EarthDipole(), len(idx), max_rows=256, max_switch=32)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.02, per_tracer_launches=int(len(idx) < n))
        ens.set_particles(w["pos"][idx], vel[idx], 0.0, mass[idx], charge[idx])
        ens.upload()
        ens.adaptive_init()
        st = ens.advance("adaptive", 0.5)
        h = ens.download()
        if len(idx) == n:
            assert st["accepted"] == h["naccept"].sum() and st["switches"] == h["nswitch"].sum() and st["launches"] == 1
            assert (h["status"] == 0).sum() > n - 400
        out.append([h[a].copy() for a in ("s", "t_row", "tcur", "mu", "status", "mode", "naccept", "nreject", "nfcn", "nswitch")])
    assert out[1][-1].sum() > 10
    for a, b in zip(*out):
        assert np.array_equal(a[..., :: n // 300], b, equal_nan=a.dtype.kind == "f")
