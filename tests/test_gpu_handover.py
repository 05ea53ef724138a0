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
