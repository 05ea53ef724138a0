"""RKF45 over more tracers than a launch has lanes: a lane that has finished its tracer
takes no part in the attempt that its warp goes on to make. Every tracer is advanced,
and to the state of a small ensemble."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["gc", "particle"])
def test_lanes_released_between_intervals(kind):
    from rapt_gb300 import Ensemble
    n = 90000
    w = W.config2(n, seed=23) if kind == "gc" else W.config4(n, 23)
    delta = np.random.default_rng(8).choice([0.01, 0.03], n) if kind == "gc" else w["delta"] * 0.004
    out = []
    which = np.random.default_rng(9).choice(n, 500, replace=False)
    for idx in (np.arange(n), which):
        u = W.subsample(w, idx)
        ens = Ensemble(F.DoubleDipole() if kind == "gc" else F.EarthDipole(), len(idx), max_rows=16)
        ens.configure(rtol=1e-7, atol=1e-7, gctimestep=0.01, cyclotronresolution=10, tableau=1)
        if kind == "gc":
            ens.set_guiding_centers(u["pos"], u["v"], pa=u["pa"], t0=0.5, mass=u["mass"], charge=u["charge"])
        else:
            ens.set_particles(u["pos"], u["vel"], 0.5, u["mass"], u["charge"])
        ens.upload()
        st = ens.advance(kind, delta[idx])
        h = ens.download()
        assert st["done"] == len(idx) and (h["naccept"] > 0).all()
        rows, _, nrows, _, _ = ens.rows()
        rows = np.where(np.arange(16)[None, :, None] < nrows[:, None, None], rows, 0.0)
        out.append([h[a].copy() for a in ("s", "t_row", "tcur", "status", "naccept", "nreject", "nfcn")] + [nrows, rows])
    for a, b in zip(*out):
        a = a[which] if a.ndim != 2 else a[:, which]
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
