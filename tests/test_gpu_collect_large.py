"""Sample collection in the FP32 forms over ensembles that fill the GPU: the blocks
that keep in step hold their warps' sample rows in more shared memory than a launch
gets without asking (from 77,825 tracers in the learned form, 116,737 without the
network), and end in the states and samples of small blocks."""
import numpy as np
import pytest

from rapt_gb300 import workloads as W
from tests._util import gpu_ensemble
from tests.test_mlp_oracle import _problem

pytestmark = pytest.mark.gpu


def _run(ctx, w, form, **cfg):
    ctx.mlp_samples_reserve(1 << 21, 3)
    ens = gpu_ensemble(w, "gc", max_rows=8, form=form, gctimestep=0.1, **cfg)
    st = ens.advance("gc", 0.1)
    ctx.mlp_samples_sort()
    h = ens.download()
    out = [h[a].copy() for a in ("s", "t_row", "status", "naccept", "nreject", "nfcn")]
    if cfg.get("collect"):
        out.append(ctx.mlp_samples_download())
    return st, out


@pytest.mark.parametrize("form,n", [(1, 116736), (1, 116737), (1, 155648), (3, 77825), (3, 120001), (3, 170000)])
def test_collecting_in_large_blocks(ctx, form, n):
    if form == 3:
        ctx.mlp_set_params(_problem(5, n=64)[0])
    w = W.config2(n, seed=21)
    st, a = _run(ctx, w, form, collect=1)
    _, b = _run(ctx, w, form, collect=1, threads_per_block=128)
    _, plain = _run(ctx, w, form)
    assert st["done"] == n and 0 < len(a[-1]) < 1 << 21
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
    for x, y in zip(a, plain):
        assert np.array_equal(x, y)
