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
