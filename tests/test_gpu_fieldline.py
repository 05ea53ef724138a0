"""Field-line integrals at the edges of their range: lines of three to a few
hundred points (the equatorial closed form, the shortest splines, long lines),
and teams of bounce centres that end at different times in one warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Re = 6378137.0
# the oracle's 8-node quadrature of the same spline is up to 3.5e-10 off its
# closed form (asymmetric wells, long double arithmetic)
TOL = 1e-9


@pytest.mark.parametrize("model", ["EarthDipole", "DoubleDipole"])
@pytest.mark.parametrize("pa", [5.0, 20.0, 60.0, 84.0, 87.5, 88.5, 89.3, 89.9])
def test_paths_and_invariants_from_short_to_long_lines(ctx, oracle, model, pa):
    from rapt_gb300 import fields as F
    fld = getattr(F, model)()
    fld.bind(ctx)
    ctx.set_config()
    f = oracle.field(model)
    tpos = np.array([[0.0, L * Re * np.cos(ph), L * Re * np.sin(ph), 0.0] for L in (4.0, 5.3, 6.7)
                     for ph in (0.1, 2.0, 4.4)])
    Bm = np.asarray(fld.magB(tpos)) / np.sin(np.radians(pa)) ** 2
    for what, ref in (("halfbouncepath", lambda p, b: oracle.halfbouncepath(f, p, b, quad=1)[0]),
                      ("eye", lambda p, b: oracle.eye(f, p, b, quad=1))):
        got = ctx.bc_eval(what, tpos, Bm, 0.03 * Re)[:, 0]
        want = np.array([ref(p, b) for p, b in zip(tpos, Bm)])
        assert np.array_equal(np.isnan(got), np.isnan(want))
        ok = np.isfinite(want)
        assert np.all(np.abs(got - want)[ok] <= TOL * np.abs(want[ok])), (what, pa, got, want)


@pytest.mark.parametrize("n", [1, 2, 5, 9])
def test_bounce_center_teams(ctx, oracle, n):
    """Rows of n bounce centres of different periods and pitch angles (different
    step counts in one warp, idle teams at the end) against the oracle's, and
    against each advanced alone."""
    from rapt_gb300 import fields as F
    from rapt_gb300 import workloads as W
    w = W.bc_drift(n, seed=3)
    fld = F.DoubleDipole()
    fld.bind(ctx)
    ctx.set_config(rtol=1.49012e-8, atol=1.49012e-8)
    f = oracle.field("DoubleDipole")
    cfg = oracle.config(rtol=1.49012e-8, atol=1.49012e-8)
    tpos = np.column_stack([np.zeros(n), w["pos"]])
    g = 1 / np.sqrt(1 - (w["v"] / W.c) ** 2)
    fld.bind(ctx)
    B = np.array([np.linalg.norm(b[:3]) for b in ctx.field_eval("B", tpos)])
    mu = (g * w["v"] * np.sin(np.radians(w["eqpa"]))) ** 2 * w["mass"] / (2 * B)
    st = np.column_stack([tpos, np.zeros(n)])
    cst = np.column_stack([w["v"], mu, w["mass"], w["charge"]])
    end, rows, nr, status, _ = ctx.bc_advance(st.copy(), cst, 1.0, 0.1, 0.03 * Re, 16)
    assert np.all(status == 0)
    for i in range(n):
        s, orows, _ = oracle.bc_advance(f, cfg, st[i].copy(), *cst[i], 1.0, 0.1, 0.03 * Re, quad=1)
        assert s == 0 and nr[i] == len(orows)
        assert np.allclose(rows[i, :nr[i]], orows, rtol=TOL, atol=TOL * Re)
        one, rows1, nr1, _, _ = ctx.bc_advance(st[i:i + 1].copy(), cst[i:i + 1], 1.0, 0.1, 0.03 * Re, 16)
        assert nr1[0] == nr[i] and np.array_equal(rows1[0, :nr[i]], rows[i, :nr[i]]) and np.array_equal(one[0], end[i])
