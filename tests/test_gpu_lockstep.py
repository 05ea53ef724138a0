"""FP32-form guiding centres in large blocks whose warps keep in step end in the same
bits as in small blocks, whatever the fill of the last block or of a launch's end."""
import numpy as np
import pytest

from rapt_gb300 import fields as F
from rapt_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _run(n, w, delta, field=F.DoubleDipole, **cfg):
    from rapt_gb300 import Ensemble
    ens = Ensemble(field(), n, max_rows=24)
    ens.configure(rtol=1e-7, atol=1e-7, form=1, **cfg)
    ens.set_guiding_centers(w["pos"][:n], w["v"][:n], pa=w["pa"][:n], t0=0.5, mass=w["mass"][:n], charge=w["charge"][:n])
    ens.upload()
    ens.advance("gc", delta[:n])
    h = ens.download()
    return [h[a][..., :n].copy() for a in ("s", "t_row", "mu", "status", "naccept", "nreject", "nfcn")] + [ens.rows()[2][:n].copy()]


# one tracer; one warp an SM group; 512 threads, the smallest that keep in step, and a
# ragged last block; 896 threads; full blocks and a second wave
@pytest.mark.parametrize("n", [1, 4864, 58500, 77825, 130001, 155648, 190000])
@pytest.mark.parametrize("cfg", [{"gctimestep": 0.02}, {"gctimestep": 0.02, "max_steps_per_launch": 5}])
def test_block_sizes(n, cfg):
    w = W.config2(n, seed=7)
    delta = np.random.default_rng(3).choice([0.0, 0.02, 0.05], n)
    a = _run(n, w, delta, **cfg)
    b = _run(n, w, delta, threads_per_block=128, **cfg)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")


def test_bounce_cadence():
    n = 60000
    w = W.config2(n, seed=8)
    delta = np.full(n, 0.02)
    cfg = dict(gctimestep=0.0, bounceresolution=20.0)
    for x, y in zip(_run(n, w, delta, **cfg), _run(n, w, delta, threads_per_block=128, **cfg)):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
