// fieldline.cuh -- the guiding-centre bounce period on the device: the output
// cadence of GuidingCenter.advance when params["GCtimestep"] == 0
// (rapt/GuidingCenter.py:443-446: dt = bounceperiod() / bounceresolution).
//
// One thread computes one tracer's bounce period, once per advance() call
// (and per Adaptive guiding-centre segment), following
//   GuidingCenter.bounceperiod      rapt/GuidingCenter.py:593-606
//   flutils.halfbouncepath          rapt/flutils.py:254-316
//   Fieldline.trace with rkf        rapt/fieldline.py:13-107, rapt/rkf.py:13-143
// and the SciPy routines halfbouncepath calls, from their published methods:
// the quadratic interpolating B-spline of interp1d(kind='quadratic'), its
// mirror points (the panels' roots; Brent's method where the line is not one
// well) and the integral between them, taken exactly where the reference calls
// quad (fl_well; fl_bounce_integral for the other lines).
//
// The (s, |B|) samples of the trace live in a per-thread scratch buffer:
// the backward half written downwards from slot cap, the forward half upwards,
// so the joined curve is contiguous. The spline solve reuses the buffer.
#pragma once
#include <cfloat>

#include "fields.cuh"

namespace rapt {

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
// numpy's 3-vector dot rounds as fma(a2, b2, fma(a1, b1, a0 b0))
__device__ __forceinline__ double ndot3(const double* a, const double* b) {
  return __fma_rn(a[2], b[2], __fma_rn(a[1], b[1], __dmul_rn(a[0], b[0])));
}

template <int M>
__device__ __forceinline__ double fl_magB(const FieldP& f, double t, double x, double y, double z) {
  double B[3];
  Field<M>::B(f, t, x, y, z, B);
  return sqrt(ndot3(B, B));
}

// _Field.curvature (fields.py:155-174) with _Field.gradB (fields.py:111-131);
// np.dot(gB, |B|) is elementwise there (kept).
template <int M>
__device__ double fl_curvature(const FieldP& f, double t, const double* X) {
  double Bv[3];
  Field<M>::B(f, t, X[0], X[1], X[2], Bv);
  const double B = sqrt(ndot3(Bv, Bv));
  const double d = f.gradstep;
  double gp[3];
#pragma unroll 1
  for (int i = 0; i < 3; ++i) {
    double xp[3] = {X[0], X[1], X[2]}, xm[3] = {X[0], X[1], X[2]};
    xp[i] = da(X[i], d);
    xm[i] = da(X[i], -d);
    const double g = (fl_magB<M>(f, t, xp[0], xp[1], xp[2]) - fl_magB<M>(f, t, xm[0], xm[1], xm[2])) / (2 * d);
    gp[i] = da(g, -dm(dm(g, B) / dm(B, B), Bv[i]));
  }
  return sqrt(ndot3(gp, gp)) / B;
}

// One direction of Fieldline.trace (fieldline.py:53-105): repeated rkf(f, 0, ds,
// x0, tol, hmax = ds, hmin = 1e-6) calls (rkf.py:13-143) along sign b from X
// until |B| > Bm. Accepted points go to slots idx, idx + dirn, ... (arc length
// and |B|); where rkf raises, the reference keeps none of that call's points
// (fieldline.py:68-69) and the trace ends. overflow: the buffer is full, or the
// field is not finite (the caller's answer is NaN either way).
//
// Every stored value is the reference's bit for bit (products and sums rounded
// separately, quotients by |B|): the second invariant's differences, and the
// step sizes chosen on them, see the trace's last bits. What the reference's
// arithmetic repeats is formed once: an accepted point's field is also the next
// step's first stage; the arc length's slope is +-1 and its error estimate
// zero; the step factor 0.84 (tol / r)^(1/4), which the cap hmax cuts off as
// long as r is under about half of tol, is evaluated only where it can matter.
template <int M>
__device__ __forceinline__ void fl_unit(const FieldP& f, double t, const double* X, double* u, double& mag) {
  double B[3];
  Field<M>::B(f, t, X[0], X[1], X[2], B);
  mag = sqrt(ndot3(B, B));
  u[0] = B[0] / mag; u[1] = B[1] / mag; u[2] = B[2] / mag;
}

template <int M>
__device__ __noinline__ int fl_trace_dir(const FieldP& f, double t0, const double* X, double Bm, double ds,
                                         bool forward, double* S, double* Bs, int cap, bool& overflow) {
  constexpr double b21 = 2.500000000000000e-01, b31 = 9.375000000000000e-02, b32 = 2.812500000000000e-01,
                   b41 = 8.793809740555303e-01, b42 = -3.277196176604461e+00, b43 = 3.320892125625853e+00,
                   b51 = 2.032407407407407e+00, b52 = -8.000000000000000e+00, b53 = 7.173489278752436e+00,
                   b54 = -2.058966861598441e-01, b61 = -2.962962962962963e-01, b62 = 2.000000000000000e+00,
                   b63 = -1.381676413255361e+00, b64 = 4.529727095516569e-01, b65 = -2.750000000000000e-01;
  constexpr double r1 = 2.777777777777778e-03, r3 = -2.994152046783626e-02, r4 = -2.919989367357789e-02,
                   r5 = 2.000000000000000e-02, r6 = 3.636363636363636e-02;
  constexpr double c1 = 1.157407407407407e-01, c3 = 5.489278752436647e-01, c4 = 5.353313840155945e-01,
                   c5 = -2.000000000000000e-01;
  constexpr double hmin = 1e-6;
  constexpr double quarter = 0.4978;  // under 0.84^4: below quarter * tol the factor is above 1
  const double tol = forward ? 1e-3 : 1e-4;  // fieldline.py:67 and :92
  const int dirn = forward ? 1 : -1;
  int idx = cap;  // slot of the start point
  double x[3] = {X[0], X[1], X[2]}, u[3], mag, s = 0.0;
  fl_unit<M>(f, t0, x, u, mag);
  for (int guard = 0; guard < 4 * cap; ++guard) {
    const int before = idx;
    double t = 0.0, h = ds;
    bool raised = false;
    for (int inner = 0; inner < 100000 && t < ds; ++inner) {
      if (da(t, h) > ds) h = da(ds, -t);
      const double hs = forward ? h : -h;  // h b and h (-b) alike
      double k1[3], k2[3], k3[3], k4[3], k5[3], k6[3], xt[3], v[3], m;
#pragma unroll
      for (int i = 0; i < 3; ++i) { k1[i] = dm(hs, u[i]); xt[i] = da(x[i], dm(b21, k1[i])); }
      fl_unit<M>(f, t0, xt, v, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) { k2[i] = dm(hs, v[i]); xt[i] = da(da(x[i], dm(b31, k1[i])), dm(b32, k2[i])); }
      fl_unit<M>(f, t0, xt, v, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        k3[i] = dm(hs, v[i]);
        xt[i] = da(da(da(x[i], dm(b41, k1[i])), dm(b42, k2[i])), dm(b43, k3[i]));
      }
      fl_unit<M>(f, t0, xt, v, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        k4[i] = dm(hs, v[i]);
        xt[i] = da(da(da(da(x[i], dm(b51, k1[i])), dm(b52, k2[i])), dm(b53, k3[i])), dm(b54, k4[i]));
      }
      fl_unit<M>(f, t0, xt, v, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        k5[i] = dm(hs, v[i]);
        xt[i] = da(da(da(da(da(x[i], dm(b61, k1[i])), dm(b62, k2[i])), dm(b63, k3[i])), dm(b64, k4[i])),
                   dm(b65, k5[i]));
      }
      fl_unit<M>(f, t0, xt, v, m);
      double e = 0.0;  // max_i |sum_j r_j k_j|
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        k6[i] = dm(hs, v[i]);
        e = fmax(e, fabs(da(da(da(da(dm(r1, k1[i]), dm(r3, k3[i])), dm(r4, k4[i])), dm(r5, k5[i])), dm(r6, k6[i]))));
      }
      const double r = e / h;
      if (r <= tol) {
        t = da(t, h);
        s = da(da(da(da(s, dm(c1, hs)), dm(c3, hs)), dm(c4, hs)), dm(c5, hs));
#pragma unroll
        for (int i = 0; i < 3; ++i)
          x[i] = da(da(da(da(x[i], dm(c1, k1[i])), dm(c3, k3[i])), dm(c4, k4[i])), dm(c5, k5[i]));
        idx += dirn;
        if (idx < 0 || idx > 2 * cap - 1) { overflow = true; return before; }
        fl_unit<M>(f, t0, x, u, mag);
        if (!isfinite(mag)) { overflow = true; return before; }
        S[idx] = s;
        Bs[idx] = mag;
      }
      if (h != ds || r > quarter * tol) {  // else the factor takes h above hmax, which caps it
        h = dm(h, fmin(fmax(dm(0.84, pow(tol / r, 0.25)), 0.1), 4.0));
        if (h > ds) h = ds;
        else if (h < hmin) { raised = true; break; }  // not asked of a capped step (ds may be below hmin)
      }
    }
    if (raised) return before;
    if (mag > Bm) break;
  }
  return idx;
}

// ---------------------------------------------------------------- quadratic spline
// Interpolating B-spline of degree 2 on n points x[0..n-1] (knots x0 x0 x0,
// midpoints of (x1,x2) .. (x_{n-3},x_{n-2}), x_{n-1} x3); c[0..n-1] coefficients.
struct DSpline2 {
  const double* x;
  const double* c;
  int n;
  __device__ __forceinline__ double knot(int j) const {
    return j <= 2 ? x[0] : (j >= n ? x[n - 1] : (x[j - 2] + x[j - 1]) / 2.0);
  }
  __device__ __forceinline__ int find(double v) const {
    if (v >= knot(n)) return n - 1;
    int lo = 2, hi = n;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (v < knot(mid)) hi = mid; else lo = mid;
    }
    return lo;
  }
  __device__ __forceinline__ void basis(double v, int l, double* h) const {
    double hh[2];
    h[0] = 1.0;
    h[1] = h[2] = 0.0;
#pragma unroll
    for (int j = 1; j <= 2; ++j) {
      for (int i = 0; i < j; ++i) hh[i] = h[i];
      h[0] = 0.0;
      for (int m = 1; m <= j; ++m) {
        const double xb = knot(l + m), xa = knot(l + m - j);
        if (xb == xa) { h[m] = 0.0; continue; }
        const double w = hh[m - 1] / (xb - xa);
        h[m - 1] = da(h[m - 1], dm(w, xb - v));
        h[m] = dm(w, v - xa);
      }
    }
  }
  __device__ __forceinline__ double operator()(double v) const { return on(v, find(v)); }
  // the value at v on panel l
  __device__ __forceinline__ double on(double v, int l) const {
    double h[3];
    basis(v, l, h);
    double y = 0.0;
    for (int a = 0; a <= 2; ++a) y = da(y, dm(c[l + a - 2], h[a]));
    return y;
  }
};

// Collocation solve (tridiagonal: x_i lies in [t[i+1], t[i+2])), in place:
// yc holds the data on entry and the coefficients on exit; di, up scratch.
static __device__ __noinline__ void spline2_solve(const double* x, double* yc, double* di, double* up, int n) {
  DSpline2 sp{x, yc, n};
  // forward elimination row by row (the lower entry is formed when the row is built)
  for (int i = 0; i < n; ++i) {
    const int l = min(max(i + 1, 2), n - 1);  // the panel that holds x[i]
    double h[3];
    sp.basis(x[i], l, h);
    double lo = 0.0, d = 0.0, u = 0.0;
    for (int a = 0; a <= 2; ++a) {
      const int j = l + a - 2;
      if (j == i - 1) lo = h[a];
      else if (j == i) d = h[a];
      else if (j == i + 1) u = h[a];
    }
    if (i > 0) {
      const double m = lo / di[i - 1];
      d = da(d, -dm(m, up[i - 1]));
      yc[i] = da(yc[i], -dm(m, yc[i - 1]));
    }
    di[i] = d;
    up[i] = u;
  }
  yc[n - 1] = yc[n - 1] / di[n - 1];
  for (int i = n - 2; i >= 0; --i) yc[i] = da(yc[i], -dm(up[i], yc[i + 1])) / di[i];
}

// ---------------------------------------------------------------- brentq
struct MirrorFn {
  DSpline2 sp;
  double Bm;
  __device__ __forceinline__ double operator()(double v) const { return da(sp(v), -Bm); }
};

static __device__ __noinline__ double fl_brentq(const MirrorFn& f, double xa, double xb) {
  const double xtol = 2e-12, rtol = 4 * DBL_EPSILON;
  double xpre = xa, xcur = xb, xblk = 0.0, fpre, fcur, fblk = 0.0, spre = 0.0, scur = 0.0, sbis;
  fpre = f(xpre);
  fcur = f(xcur);
  if (fpre == 0) return xpre;
  if (fcur == 0) return xcur;
  for (int i = 0; i < 100; ++i) {
    if (fpre != 0 && fcur != 0 && (signbit(fpre) != signbit(fcur))) {
      xblk = xpre;
      fblk = fpre;
      spre = scur = xcur - xpre;
    }
    if (fabs(fblk) < fabs(fcur)) {
      xpre = xcur; xcur = xblk; xblk = xpre;
      fpre = fcur; fcur = fblk; fblk = fpre;
    }
    const double delta = da(xtol, dm(rtol, fabs(xcur))) / 2;
    sbis = (xblk - xcur) / 2;
    if (fcur == 0 || fabs(sbis) < delta) return xcur;
    if (fabs(spre) > delta && fabs(fcur) < fabs(fpre)) {
      double stry;
      if (xpre == xblk) {
        stry = dm(-fcur, xcur - xpre) / (fcur - fpre);
      } else {
        const double dpre = (fpre - fcur) / (xpre - xcur);
        const double dblk = (fblk - fcur) / (xblk - xcur);
        stry = dm(-fcur, da(dm(fblk, dblk), -dm(fpre, dpre))) / dm(dm(dblk, dpre), fblk - fpre);
      }
      if (2 * fabs(stry) < fmin(fabs(spre), da(3 * fabs(sbis), -delta))) {
        spre = scur;
        scur = stry;
      } else {
        spre = sbis;
        scur = sbis;
      }
    } else {
      spre = sbis;
      scur = sbis;
    }
    xpre = xcur;
    fpre = fcur;
    if (fabs(scur) > delta) xcur = da(xcur, scur);
    else xcur = da(xcur, sbis > 0 ? delta : -delta);
    fcur = f(xcur);
  }
  return xcur;
}

// ---------------------------------------------------------------- half-bounce integral
// The reference integrates 1/sqrt(1 - B(s)/Bm) over [sm1, sm2] with QUADPACK
// QAGS at epsrel 1e-4; on these symmetric field lines the two mirror-point
// singularities give tied error estimates and QAGS's bisection order (and its
// result, to ~5e-6) depends on the last bit of the spline values. Here the
// same spline is integrated to convergence instead: s = c + h sin(theta)
// removes the singularities and an 8-point Gauss-Legendre rule runs on every
// panel between the images of the spline's knots.
static __device__ __noinline__ void gauss_legendre8(double* x, double* w) {
  const int n = 8;
  for (int i = 0; i < n / 2; ++i) {
    double z = cos(kPi * (i + 0.75) / (n + 0.5)), pp = 0.0;
    for (int it = 0; it < 100; ++it) {
      double p1 = 1.0, p2 = 0.0;
      for (int j = 1; j <= n; ++j) {
        const double p3 = p2;
        p2 = p1;
        p1 = da(dm(dm(2.0 * j - 1.0, z), p2), -dm(j - 1.0, p3)) / j;
      }
      pp = dm(n, da(dm(z, p1), -p2)) / da(dm(z, z), -1.0);
      const double z1 = z;
      z = da(z1, -(p1 / pp));
      if (fabs(z - z1) <= 1e-16) break;
    }
    x[i] = -z;
    x[n - 1 - i] = z;
    w[i] = w[n - 1 - i] = 2.0 / dm(dm(da(1.0, -dm(z, z)), pp), pp);
  }
}

// inv: integrand 1/sqrt(1 - B/Bm) (half-bounce path); otherwise sqrt(1 - B/Bm)
// (the second invariant I), which the substitution leaves smooth as well.
// Panel edges in theta: -pi/2, the knots j0 .. j1 inside (sm1, sm2), pi/2.
struct FlPanels {
  double c, h;
  int j0, count;  // first knot inside; panels
};
__device__ __forceinline__ FlPanels fl_panels(const DSpline2& sp, double sm1, double sm2) {
  FlPanels P{dm(0.5, da(sm1, sm2)), dm(0.5, da(sm2, -sm1)), 0, 1};
  for (int j = 3; j < sp.n; ++j) {
    const double tj = sp.knot(j);
    if (!(tj > sm1 && tj < sm2)) continue;
    if (P.count == 1) P.j0 = j;
    ++P.count;
  }
  return P;
}
__device__ __forceinline__ double fl_panel_edge(const DSpline2& sp, const FlPanels& P, int q) {
  if (q == 0) return -kPi / 2;
  return q == P.count ? kPi / 2 : asin((sp.knot(P.j0 + q - 1) - P.c) / P.h);
}
// One panel between its edges ea, eb: 8 nodes gx, weights gw. The spline panel
// is the knots' own (found by search only where no knot lies inside).
static __device__ __noinline__ double fl_panel_sum(const DSpline2& sp, const FlPanels& P, int q, double ea, double eb,
                                                   const double* gx, const double* gw, double Bm, bool inv) {
  const double mid = dm(0.5, da(ea, eb)), half = dm(0.5, da(eb, -ea));
  const int l = P.count == 1 ? sp.find(P.c) : P.j0 + q - 1;
  double ps = 0.0;
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    const double th = da(mid, dm(half, gx[k]));
    double sn, cs;
    sincos(th, &sn, &cs);
    const double arg = da(1.0, -(sp.on(da(P.c, dm(P.h, sn)), l) / Bm));
    if (arg > 0.0) {
      const double hc = dm(P.h, cs), root = sqrt(arg);
      ps = da(ps, dm(gw[k], inv ? hc / root : dm(hc, root)));
    }
  }
  return dm(half, ps);
}
static __device__ __noinline__ double fl_bounce_integral(const DSpline2& sp, double sm1, double sm2, double Bm,
                                                         bool inv) {
  double gx[8], gw[8];
  gauss_legendre8(gx, gw);
  const FlPanels P = fl_panels(sp, sm1, sm2);
  double sum = 0.0, ea = -kPi / 2;
  for (int q = 0; q < P.count; ++q) {
    const double eb = fl_panel_edge(sp, P, q + 1);
    sum = da(sum, fl_panel_sum(sp, P, q, ea, eb, gx, gw, Bm, inv));
    ea = eb;
  }
  return sum;
}

// ---------------------------------------------------------------- the spline's integral in closed form
// On one panel 1 - B/Bm is a quadratic q(u) = A0 + A1 u + A2 u^2, and with
// ra = sqrt(q(a)), rb = sqrt(q(b)), D = b - a, w = D / (ra + rb), y = -A2 w^2,
// f(y) = atan(sqrt y) / sqrt y (atanh for y < 0), g(y) = (1 - f(y)) / y:
//   int_a^b du / sqrt(q) = 2 w f(y)
//   int_a^b sqrt(q) du   = D (ra + rb) / 4 + w (2 (ra^2 + rb^2) - A2 D^2) / 4 - w^3 disc g(y) / 4
// with disc = A1^2 - 4 A0 A2 (the elementary antiderivatives, rearranged so that
// nothing cancels as A2 goes to 0). The mirror points, where ra or rb is 0, need
// no care of their own.
__device__ __forceinline__ void fl_atan_ratio(double y, double& fy, double& gy) {
  if (fabs(y) < 0.04) {  // the alternating series of f; truncation under 1e-16
    constexpr double c[11] = {1.0 / 3,  1.0 / 5,  1.0 / 7,  1.0 / 9,  1.0 / 11, 1.0 / 13,
                              1.0 / 15, 1.0 / 17, 1.0 / 19, 1.0 / 21, 1.0 / 23};
    double p = c[10];
#pragma unroll
    for (int k = 9; k >= 0; --k) p = fma(-y, p, c[k]);
    gy = p;
    fy = fma(-y, p, 1.0);
  } else {
    const double r = sqrt(fabs(y));
    fy = (y > 0.0 ? atan(r) : atanh(r)) / r;
    gy = (1.0 - fy) / y;
  }
}

// Interpolating quadratic spline of the samples yc at x (n >= 3; yc leaves as
// the coefficients; rd, up: scratch) and the integral of 1/sqrt(1 - B/Bm) (inv)
// or sqrt(1 - B/Bm) between its mirror points. The collocation matrix is
// tridiagonal (x_i lies on panel i + 1): one forward sweep, and one backward
// sweep that integrates each panel as its coefficients appear, the mirror
// points being roots of the outermost panels' quadratics. ~85 FP64
// instructions a point, where a binary search per value, Brent's method and 8
// quadrature nodes a panel (a sine, a cosine and a spline value each) took
// ~1,700. A line that is not one well between its outermost points (no sign
// change there, or B > Bm in between) takes those routines, which skip the
// stretches above Bm. 16,384 guiding centres at the bounce-period cadence,
// advance(0.2), with the trace above: 56.0 ms before, 29.9 ms.
static __device__ __noinline__ double fl_well(const double* x, double* yc, double* rd, double* up, int n, double Bm,
                                              bool inv) {
  bool bad = !(n >= 4 && yc[0] > Bm && yc[1] <= Bm && yc[n - 2] <= Bm && yc[n - 1] > Bm);
  const double iBm = 1.0 / Bm, x0 = x[0], xl = x[n - 1];
  rd[0] = 1.0;
  up[0] = 0.0;
  {
    double T0 = x0, T1 = x0, T2 = n > 3 ? 0.5 * (x[1] + x[2]) : xl;
    double r0 = 1.0 / (T2 - T0), cp = yc[0], rdp = 1.0, upp = 0.0;
    for (int i = 1; i <= n - 2; ++i) {
      const double T3 = i + 3 >= n ? xl : 0.5 * (x[i + 1] + x[i + 2]);
      const double r1 = 1.0 / (T2 - T1), r2 = 1.0 / (T3 - T1);
      const double a = T2 - x[i], c = x[i] - T1;
      const double h0 = (a * r1) * (a * r0), h2 = (c * r1) * (c * r2);
      const double m = h0 * rdp;
      rdp = 1.0 / (1.0 - h0 - h2 - m * upp);
      upp = h2;
      cp = fma(-m, cp, yc[i]);
      rd[i] = rdp; up[i] = upp; yc[i] = cp;
      T0 = T1; T1 = T2; T2 = T3; r0 = r2;
    }
  }
  double sum = 0.0, c2 = 0.0, c1 = yc[n - 1];
  // knots T1, T2 of the panel in hand, walking down from panel n - 1
  double T2 = xl, T1 = n > 3 ? 0.5 * (x[n - 3] + x[n - 2]) : x0, r2 = 1.0 / (T2 - T1), rhi = 0.0;
  for (int i = n - 2; i >= 0; --i) {
    const double c0 = i ? fma(-up[i], c1, yc[i]) * rd[i] : yc[0];
    yc[i] = c0;
    if (i <= n - 3 && !bad) {  // panel i + 2: coefficients c0, c1, c2
      const bool left = i == 0, right = i == n - 3;
      const double T0 = i <= 1 ? x0 : 0.5 * (x[i - 1] + x[i]);
      const double D1 = T2 - T1, r1 = 1.0 / D1, r0 = 1.0 / (T2 - T0);
      const double al = (c0 - c1) * iBm * r1 * r0, be = (c2 - c1) * iBm * r1 * r2;
      const double C = fma(-c1, iBm, 1.0), A2 = -(al + be);
      const double qa = fma(-al * D1, D1, C), qb = fma(-be * D1, D1, C);
      double ua = 0.0, ub = D1, ra = 0.0, rb = rhi;
      if (right) {  // q as a quadratic in the distance from the panel's end
        const double B1 = 2.0 * be * D1, disc = fma(B1, B1, -4.0 * qb * A2);
        bad = bad || !(qb < 0.0 && disc >= 0.0);
        ub = D1 - (-2.0 * qb) / (B1 + sqrt(disc));
        rb = 0.0;
      }
      if (left) {
        const double B1 = 2.0 * al * D1, disc = fma(B1, B1, -4.0 * qa * A2);
        bad = bad || !(qa < 0.0 && disc >= 0.0);
        ua = (-2.0 * qa) / (B1 + sqrt(disc));
      } else {
        bad = bad || !(qa > 0.0);
        ra = sqrt(qa);
      }
      const double D = ub - ua, mu = fma(A2, ua + ub, 2.0 * al * D1);
      const double q2 = fma(ra, ra, rb * rb), AD = A2 * D;
      const double disc = fma(mu, mu, fma(AD, AD, -2.0 * A2 * q2));
      bad = bad || !(D > 0.0) || (A2 > 0.0 && disc >= 0.0 && fabs(mu) < AD);  // a stretch above Bm inside
      const double w = D / (ra + rb);
      double fy, gy;
      fl_atan_ratio(-A2 * w * w, fy, gy);
      if (inv) sum = fma(2.0 * w, fy, sum);
      else sum += 0.25 * fma(D, ra + rb, w * (2.0 * q2 - AD * D - w * w * disc * gy));
      rhi = ra;
      T2 = T1; T1 = T0; r2 = r0;
    }
    c2 = c1;
    c1 = c0;
  }
  if (!bad) return sum;
  const DSpline2 sp{x, yc, n};
  const MirrorFn g{sp, Bm};
  const double sm1 = fl_brentq(g, x[0], x[1]);
  const double sm2 = !inv && sp(x[n - 2]) == Bm ? x[n - 2] : fl_brentq(g, x[n - 2], x[n - 1]);
  return fl_bounce_integral(sp, sm1, sm2, Bm, inv);
}

// ---------------------------------------------------------------- half-bounce path and bounce period
// A thread's scratch: 4 * (2 * cap) doubles: arc length and |B| of the joined
// curve, then (in place of |B|) the spline coefficients, and the solve's rows.
//
// Step of the trace through X (fieldline.py:31-35) and its start sample.
template <int M>
__device__ __forceinline__ double fl_start(const FieldP& f, double t, const double* X, double flres, double* scratch,
                                           int cap) {
  const double ds = 1.0 / fl_curvature<M>(f, t, X) / flres;
  scratch[cap] = 0.0;
  scratch[3 * cap] = fl_magB<M>(f, t, X[0], X[1], X[2]);
  return ds;
}

// The samples that the integral is taken over: n from slot lo of the scratch, or
// (n == 0) the answer itself.
struct FlCut {
  int lo, n;
  double value;
};
// flutils.halfbouncepath (flutils.py:254-316) of the traced samples in slots
// first .. first + n0 - 1, mirror field Bm.
static __device__ __noinline__ FlCut fl_cut_path(const double* scratch, int cap, int first, int n0, double Bm) {
  const double* S = scratch;
  const double* Bs = scratch + 2 * cap;
  int fin = -1, lin = -1;
  for (int i = 0; i < n0; ++i)
    if (Bs[first + i] <= Bm) {
      if (fin < 0) fin = i;
      lin = i;
    }
  int i1, i2;
  if (fin < 0) { i1 = (n0 - 3) / 2; i2 = (n0 + 1) / 2; }
  else { i1 = fin - 1; i2 = lin + 1; }
  const int lo = i1 < 0 ? 0 : i1, hi = i2 > n0 - 1 ? n0 - 1 : i2;
  const int n = hi - lo + 1;
  const double* s = S + first + lo;
  const double* b = Bs + first + lo;
  if (n == 3) {  // equatorial (flutils.py:292-303)
    const double s12 = s[0] - s[1], s23 = s[1] - s[2], s13 = s[0] - s[2];
    const double B2s = 2 * da(da(dm(b[0], s23), -dm(b[1], s13)), dm(b[2], s12)) / dm(dm(s12, s13), s23);
    return FlCut{0, 0, dm(kPi, sqrt(2 * Bm / B2s))};
  }
  if (n < 3) return FlCut{0, 0, nan("")};
  return FlCut{first + lo, n, 0.0};
}

// flutils.eye (flutils.py:65-151) of the traced samples: 0 where the line's
// minimum |B| exceeds Bm or equals it (equatorial); the points with B < Bm plus
// one beyond each end. The reference takes this spline branch at equatorial
// pitch angles of 70 degrees and above; below, its Simpson branch calls an
// undefined name and raises, and here the spline branch serves every pitch
// angle. NaN where the trimmed line fails the reference's assert.
static __device__ __noinline__ FlCut fl_cut_eye(const double* scratch, int cap, int first, int n0, double Bm) {
  const double* Bs = scratch + 2 * cap;
  if (n0 < 1) return FlCut{0, 0, nan("")};
  double Bmin = Bs[first];
  int fin = -1, lin = -1;
  for (int i = 0; i < n0; ++i) {
    const double v = Bs[first + i];
    Bmin = fmin(Bmin, v);
    if (v < Bm) {
      if (fin < 0) fin = i;
      lin = i;
    }
  }
  if (Bmin > Bm) return FlCut{0, 0, 0.0};
  if (fabs(Bmin - Bm) / Bm < 1e-12) return FlCut{0, 0, 0.0};
  const int lo = fin - 1 < 0 ? 0 : fin - 1, hi = lin + 1 > n0 - 1 ? n0 - 1 : lin + 1;
  const int n = hi - lo + 1;
  const double* b = Bs + first + lo;
  if (!(n >= 3 && b[0] > Bm && b[1] < Bm && b[n - 2] < Bm && b[n - 1] > Bm)) return FlCut{0, 0, nan("")};
  return FlCut{first + lo, n, 0.0};
}

__device__ __forceinline__ double fl_integral_of(double* scratch, int cap, const FlCut& cut, double Bm, bool inv) {
  if (cut.n == 0) return cut.value;
  return fl_well(scratch + cut.lo, scratch + 2 * cap + cut.lo, scratch + 4 * cap, scratch + 6 * cap, cut.n, Bm, inv);
}

// Both directions of the line through X by one thread; false where the trace
// overflows the buffer or the step is not finite.
template <int M>
__device__ bool fl_trace(const FieldP& f, double t, const double* X, double Bm, double flres, double* scratch,
                         int cap, int& first, int& n0) {
  const double ds = fl_start<M>(f, t, X, flres, scratch, cap);
  if (!(ds > 0) || !isfinite(ds)) return false;
  bool overflow = false;
  const int ifw = fl_trace_dir<M>(f, t, X, Bm, ds, true, scratch, scratch + 2 * cap, cap, overflow);
  first = fl_trace_dir<M>(f, t, X, Bm, ds, false, scratch, scratch + 2 * cap, cap, overflow);
  n0 = ifw - first + 1;
  return !overflow;
}

template <int M>
__device__ __noinline__ double fl_halfbouncepath(const FieldP& f, double t, const double* X, double Bm,
                                                 double flres, double* scratch, int cap) {
  int first, n0;
  if (!fl_trace<M>(f, t, X, Bm, flres, scratch, cap, first, n0)) return nan("");
  return fl_integral_of(scratch, cap, fl_cut_path(scratch, cap, first, n0, Bm), Bm, true);
}

template <int M>
__device__ __noinline__ double fl_eye(const FieldP& f, double t, const double* X, double Bm, double flres,
                                     double* scratch, int cap) {
  int first, n0;
  if (!fl_trace<M>(f, t, X, Bm, flres, scratch, cap, first, n0)) return nan("");
  return fl_integral_of(scratch, cap, fl_cut_eye(scratch, cap, first, n0, Bm), Bm, false);
}

// flutils.gradI (flutils.py:153-229): central differences of I over d in the
// two directions perpendicular to b built from (x, y, 0); one-sided where one
// end has I = 0. v: the two directions.
template <int M>
__device__ __forceinline__ void fl_gradI_axes(const FieldP& f, double t, const double* X, double v[2][3]) {
  const double sc = fmax(fabs(X[0]), fabs(X[1]));
  double* r = v[0];
  r[0] = X[0] / sc; r[1] = X[1] / sc; r[2] = 0.0 / sc;
  double b[3], mag;
  unit_and_mag<M>(f, t, X[0], X[1], X[2], b, mag);
  const double rb = ndot3(r, b);
  for (int i = 0; i < 3; ++i) r[i] = da(r[i], -dm(rb, b[i]));
  const double rn = sqrt(ndot3(r, r));
  for (int i = 0; i < 3; ++i) r[i] = r[i] / rn;
  v[1][0] = da(dm(b[1], r[2]), -dm(b[2], r[1]));
  v[1][1] = da(dm(b[2], r[0]), -dm(b[0], r[2]));
  v[1][2] = da(dm(b[0], r[1]), -dm(b[1], r[0]));
}
// One difference quotient from I at X + d v, X - d v and X.
__device__ __forceinline__ double fl_gradI_quotient(double Ip, double Im, double I0, double d) {
  if (Ip == 0.0) return da(I0, -Im) / d;
  if (Im == 0.0) return da(Ip, -I0) / d;
  return da(Ip, -Im) / (2.0 * d);
}
template <int M>
__device__ void fl_gradI(const FieldP& f, double t, const double* X, double Bm, double d, double flres,
                         double* scratch, int cap, double* out) {
  double v[2][3], dI[2];
  fl_gradI_axes<M>(f, t, X, v);
  for (int k = 0; k < 2; ++k) {
    const double xp[3] = {da(X[0], dm(d, v[k][0])), da(X[1], dm(d, v[k][1])), da(X[2], dm(d, v[k][2]))};
    const double xm[3] = {da(X[0], -dm(d, v[k][0])), da(X[1], -dm(d, v[k][1])), da(X[2], -dm(d, v[k][2]))};
    const double I1 = fl_eye<M>(f, t, xp, Bm, flres, scratch, cap);
    const double I2 = fl_eye<M>(f, t, xm, Bm, flres, scratch, cap);
    const double I0 = I1 == 0.0 || I2 == 0.0 ? fl_eye<M>(f, t, X, Bm, flres, scratch, cap) : 0.0;
    dI[k] = fl_gradI_quotient(I1, I2, I0, d);
  }
  for (int i = 0; i < 3; ++i) out[i] = da(dm(dI[0], v[0][i]), dm(dI[1], v[1][i]));
}

// GuidingCenter.bounceperiod (GuidingCenter.py:593-606) at state (x, y, z, ppar).
template <int M>
__device__ double gc_bounceperiod(const FieldP& f, double t, const double* y, double mu, double m, double flres,
                                  double* scratch, int cap) {
  const double Bmag = fl_magB<M>(f, t, y[0], y[1], y[2]);
  const double ppar = y[3];
  const double gamma = sqrt(da(da(1.0, dm(2.0, dm(mu, Bmag)) / dm(m, dm(kC, kC))), dm(ppar / (m * kC), ppar / (m * kC))));
  double p, v, Bmirror;
  if (gamma - 1 < 1e-6) {
    p = sqrt(da(dm(dm(2.0, m), dm(mu, Bmag)), dm(ppar, ppar)));
    v = p / m;
    Bmirror = dm(p, p) / dm(dm(2.0, m), mu);
  } else {
    p = dm(dm(m, kC), sqrt(dm(gamma + 1, gamma - 1)));
    Bmirror = dm(dm(p, p) / dm(p - ppar, p + ppar), Bmag);
    v = p / m / gamma;
  }
  return dm(2.0 / v, fl_halfbouncepath<M>(f, t, y, Bmirror, flres, scratch, cap));
}

}  // namespace rapt
