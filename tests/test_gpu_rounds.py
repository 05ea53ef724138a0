"""Adaptive ensembles that go by rounds of two kernels side by side (the FP32 form, RKF45,
dense output, step budgets, sample collection): results do not depend on how the rounds
share the GPU between the kernels, whether one mode has all tracers or both have some."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FORMS = {"fp32": {"form": 1}, "rkf": {"tableau": 1}, "dense": {"dense_output": 1}, "budget": {"max_steps_per_launch": 400}}


def _workload(modes, n):
    w = W.config4(n, 17)
    if modes == "gc":  # electrons far below the adiabatic limit
        rng = np.random.default_rng(2)
        d = w["vel"] / np.linalg.norm(w["vel"], axis=1)[:, None]
        return dict(w, vel=d * W.speed_from_ke(10 ** rng.uniform(4, 6, n), W.m_el)[:, None], mass=np.full(n, W.m_el),
                    charge=np.full(n, -W.e)), {}
    if modes == "particles":  # nothing counts as adiabatic
        return w, {"epss": 1e-9, "epst": 1e-9}
    return W.config5(n, 18), {}


def _run(modes, which, n, delta, cfg):
    from rapt_gb300 import Ensemble
    w, eps = _workload(modes, n)
    w = W.subsample(w, which)
    ens = Ensemble(F.CompressedDipole() if modes == "both" else F.DoubleDipole(), len(which), max_rows=32, max_switch=8)
    ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.05, cyclotronresolution=10, **eps, **cfg)
    ens.set_particles(w["pos"], w["vel"], 0.0, w["mass"], w["charge"])
    ens.upload()
    ens.adaptive_init()
    start = ens.download()["mode"].mean()
    st = ens.advance("adaptive", delta if delta else 0.04 * w["delta"])  # two gyro-periods, 20 rows
    h = ens.download()
    return start, st, [h[a].copy() for a in ("s", "t_row", "tcur", "mu", "status", "flags", "mode", "naccept", "nreject", "nfcn", "nswitch")]


@pytest.mark.parametrize("form", list(FORMS))
# more tracers than four times the lanes of half the GPU (one mode takes it all), and fewer
@pytest.mark.parametrize("modes,n,delta", [("gc", 120000, 0.1), ("gc", 30000, 0.1), ("particles", 90000, None), ("both", 40000, 0.1)])
def test_rounds(form, modes, n, delta):
    if form == "rkf" and modes == "both":
        delta *= 0.1
    cfg = FORMS[form]
    start, st, a = _run(modes, np.arange(n), n, delta, cfg)
    assert {"gc": start == 1, "particles": start == 0, "both": 0 < start < 1}[modes]
    assert st["done"] == n and (a[7] > 0).all()
    which = np.random.default_rng(6).choice(n, 300, replace=False)
    _, _, b = _run(modes, which, n, delta, cfg)
    for x, y in zip(a, b):
        assert np.array_equal(x[..., which], y, equal_nan=x.dtype.kind == "f")
