"""Field lines of any size: the trace's step is a fiftieth of the radius of curvature,
which rkf's hmin (1e-6) does not bound as long as the step grows, so a line of a
small dipole is the scaled line of a large one (rkf.py:118-122: hmax first)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Re = 6378137.0


def _lines(ctx, scale, pa):
    from rapt_gb300 import fields as F
    fld = F.EarthDipole()
    fld.gradientstepsize = Re * 2.0 ** -10 * scale
    fld.bind(ctx)
    ctx.set_config()
    tpos = np.array([[0.0, 5 * Re * np.cos(ph) * scale, 5 * Re * np.sin(ph) * scale, 0.0] for ph in (0.1, 2.0, 4.4)])
    Bm = np.asarray(fld.magB(tpos)) / np.sin(np.radians(pa)) ** 2
    fld.bind(ctx)
    return tpos, Bm, [ctx.bc_eval(what, tpos, Bm, 0.03 * Re * scale)[:, 0] / scale for what in ("halfbouncepath", "eye")]


@pytest.mark.parametrize("shift", [30, 37, 38, 44])  # steps of 2e-4, 1.5e-6, 8e-7 and 1.2e-8 m
@pytest.mark.parametrize("pa", [60.0, 85.0])
def test_lines_scale(ctx, oracle, shift, pa):
    """The scale is a power of two, so the scaled line's arithmetic is the large one's."""
    tpos, Bm, want = _lines(ctx, 1.0, pa)
    _, _, got = _lines(ctx, 2.0 ** -shift, pa)
    for g, w in zip(got, want):
        assert np.isfinite(w).all() and np.all(np.abs(g - w) <= 1e-12 * w)
    # the oracle keeps as many points whatever the size
    n = []
    for scale in (1.0, 2.0 ** -shift):
        f = oracle.field("EarthDipole")
        f.gradstep = Re * 2.0 ** -10 * scale
        n.append([oracle.halfbouncepath(f, p * scale, b / scale ** 3, quad=1)[1] for p, b in zip(tpos, Bm)])
    assert n[0] == n[1]
