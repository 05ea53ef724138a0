// bc_kernels.cuh -- BounceCenter (rapt/BounceCenter.py) on the device: the
// bounce-averaged drift of a guiding centre in a static magnetic field,
//   dx/dt = gamma m v^2 / (q S_b |B|^2) (grad I x B)        BounceCenter.py:236-245
// with S_b the half-bounce path (flutils.halfbouncepath) and grad I the
// gradient of the second invariant (flutils.gradI): six field-line traces per
// right-hand side.
// advance(delta) (BounceCenter.py:214-252) outputs every BCtimestep x the
// bounce period at the start, restarting DOPRI5 (SciPy's dopri5 defaults) per
// row; the host launches one interval of every tracer per kernel.
//
// The reference's isequatorial branch (BounceCenter.py:238-239) hands the
// 3-vector state to _v_grad as (t, x, y, z) and fails; it is not built.
#pragma once
#include "fieldline.cuh"
#include "steppers.cuh"
#include "tracer_kernels.cuh"

namespace rapt {

__device__ __forceinline__ void bc_drift(double kdrift, double Sb, const double* B, const double* gI, double* o) {
  const double k = kdrift / dm(Sb, ndot3(B, B));
  o[0] = dm(k, da(dm(gI[1], B[2]), -dm(gI[2], B[1])));
  o[1] = dm(k, da(dm(gI[2], B[0]), -dm(gI[0], B[2])));
  o[2] = dm(k, da(dm(gI[0], B[1]), -dm(gI[1], B[0])));
}

// The drift by one thread (single evaluations, k_bc_eval).
template <int M>
struct BcRHS {
  FieldP f;
  double Bm, kdrift, d, flres;  // kdrift = gamma m v^2 / q
  double* scratch;
  int cap;
  __device__ void operator()(double t, const double* Y, double* o) const {
    double B[3], gI[3];
    Field<M>::B(f, t, Y[0], Y[1], Y[2], B);
    const double Sb = fl_halfbouncepath<M>(f, t, Y, Bm, flres, scratch, cap);
    fl_gradI<M>(f, t, Y, Bm, d, flres, scratch, cap, gI);
    bc_drift(kdrift, Sb, B, gI, o);
  }
};

// The drift by a team of 16 lanes, called by whole warps: lane pairs trace the
// six lines -- 0: through X for the half-bounce path, 1..4: through the ends of
// the two differences, 5: through X for the one-sided differences -- one lane
// forward, one backward, into a scratch slot per line; the pair then shares the
// mirror points and the integral. All lanes return the same drift.
//
// A right-hand side is a serial chain of RKF45 steps along each line (an FP64
// instruction holds the sub-partition's FP64 pipe for 64 cycles whatever the
// number of active lanes), so the chain is what has to be short: twelve traces
// side by side instead of one after another, and no search or node table in the
// integral. The values are those of one thread doing it all, bit for bit: a
// bounce centre starts with a coordinate at 0, whose tolerance is atol alone
// (1.5e-8 m), and there the step sizes follow the drift's last bits -- which is
// also why this integral keeps its quadrature (fl_panel_sum) where the single
// evaluations take the closed form (fl_well).
// State and result go by value, in registers, as in the other right-hand sides.
// 2,048 bounce centres, advance(0.2): 682 ms with a thread a tracer, 78 ms so.
constexpr int kBcTeam = 16, kBcLines = 6;  // bc_trace_slots (launch.h) counts kBcLines slots a team
template <int M>
struct BcTeamRHS {
  const FieldP& f;
  double Bm, kdrift, d, flres;
  double* scratch;  // kBcLines slots of stride doubles
  long long stride;
  int cap;
  const double* gauss;  // the 8-point Gauss-Legendre nodes, then the weights
  bool* bad;            // set where a value is not finite
  struct D3 {
    double v0, v1, v2;
  };
  __device__ __forceinline__ void operator()(double t, const double* Y, double* o) const {
    const D3 r = eval(t, D3{Y[0], Y[1], Y[2]});
    o[0] = r.v0; o[1] = r.v1; o[2] = r.v2;
  }
  __device__ __noinline__ D3 eval(double t, D3 Yv) const {
    const double Y[3] = {Yv.v0, Yv.v1, Yv.v2};
    double o[3];
    const int lane = threadIdx.x & 31, r = lane & (kBcTeam - 1), line = min(r >> 1, kBcLines - 1);
    double B[3], v[2][3];
    Field<M>::B(f, t, Y[0], Y[1], Y[2], B);
    fl_gradI_axes<M>(f, t, Y, v);
    const double side = line == 1 || line == 3 ? d : -d;
    const bool off = line >= 1 && line <= 4;
    double X[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) X[i] = off ? da(Y[i], dm(side, line <= 2 ? v[0][i] : v[1][i])) : Y[i];
    double* scr = scratch + line * stride;
    const bool forward = (r & 1) == 0;
    bool overflow = false;
    int end = cap;
    if (r < 2 * kBcLines) {
      // both lanes of a pair start from the same sample; the first writes it
      const double ds = 1.0 / fl_curvature<M>(f, t, X) / flres;
      if (forward) { scr[cap] = 0.0; scr[3 * cap] = fl_magB<M>(f, t, X[0], X[1], X[2]); }
      overflow = !(ds > 0) || !isfinite(ds);
      if (!overflow) end = fl_trace_dir<M>(f, t, X, Bm, ds, forward, scr, scr + 2 * cap, cap, overflow);
    }
    __syncwarp();
    const int other = __shfl_xor_sync(kFull, end, 1);
    const bool over = __shfl_xor_sync(kFull, (int)overflow, 1) || overflow;
    // the pair's integral: the first lane solves the spline, each lane finds one
    // mirror point and sums half of the panels
    const int first = forward ? other : end, n0 = (forward ? end : other) - first + 1;
    const bool inv = line == 0, mine = r < 2 * kBcLines && !over;
    FlCut cut{0, 0, nan("")};
    if (mine) cut = inv ? fl_cut_path(scr, cap, first, n0, Bm) : fl_cut_eye(scr, cap, first, n0, Bm);
    __syncwarp();
    const bool need = mine && cut.n > 0;
    const DSpline2 sp{scr + cut.lo, scr + 2 * cap + cut.lo, cut.n};
    double* part = scr + 6 * cap;  // panel sums (the solve's row storage, free by then)
    if (need && forward) spline2_solve(sp.x, scr + 2 * cap + cut.lo, scr + 4 * cap, part, cut.n);
    __syncwarp();
    double root = 0.0;
    if (need) {
      const MirrorFn g{sp, Bm};
      const double e0 = forward ? sp.x[0] : sp.x[cut.n - 2], e1 = forward ? sp.x[1] : sp.x[cut.n - 1];
      root = !inv && !forward && sp(e0) == Bm ? e0 : fl_brentq(g, e0, e1);
    }
    const double sm1 = __shfl_sync(kFull, root, lane & ~1), sm2 = __shfl_sync(kFull, root, lane | 1);
    FlPanels P{};
    if (need) {
      P = fl_panels(sp, sm1, sm2);
      const int q0 = forward ? 0 : (P.count + 1) / 2, q1 = forward ? (P.count + 1) / 2 : P.count;
      double ea = q0 < q1 ? fl_panel_edge(sp, P, q0) : 0.0;
      for (int q = q0; q < q1; ++q) {
        const double eb = fl_panel_edge(sp, P, q + 1);
        part[q] = fl_panel_sum(sp, P, q, ea, eb, gauss, gauss + 8, Bm, inv);
        ea = eb;
      }
    }
    __syncwarp();
    double val = cut.value;
    if (need && forward) {
      val = 0.0;
      for (int q = 0; q < P.count; ++q) val = da(val, part[q]);
    }
    __syncwarp();
    double I[kBcLines];
#pragma unroll
    for (int k = 0; k < kBcLines; ++k) I[k] = __shfl_sync(kFull, val, (lane & ~(kBcTeam - 1)) + 2 * k);
    const bool one = I[1] == 0.0 || I[2] == 0.0 || I[3] == 0.0 || I[4] == 0.0;
    const double dI0 = fl_gradI_quotient(I[1], I[2], one ? I[5] : 0.0, d);
    const double dI1 = fl_gradI_quotient(I[3], I[4], one ? I[5] : 0.0, d);
    double gI[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gI[i] = da(dm(dI0, v[0][i]), dm(dI1, v[1][i]));
    if (!(isfinite(I[0]) && isfinite(gI[0]) && isfinite(gI[1]) && isfinite(gI[2]))) *bad = true;
    bc_drift(kdrift, I[0], B, gI, o);
    return D3{o[0], o[1], o[2]};
  }
};

__device__ __forceinline__ double bc_gamma(double v) { return 1.0 / sqrt(1.0 - (v / kC) * (v / kC)); }

// Start of advance(delta): mirror field, cadence and row count per tracer.
// st[5] = (t, x, y, z, tcur); plan[4] = (Bm, dt, K, arange step).
template <int M>
__global__ void k_bc_start(FieldP f, double flres, int64_t n, const double* st, const double* cst, double delta,
                           double bctimestep, double* plan, int32_t* status, int32_t* flag, double* scratch,
                           long long stride, int cap) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double* s = st + 5 * k;
  const double v = cst[4 * k], mu = cst[4 * k + 1], mass = cst[4 * k + 2];
  const double gamma = bc_gamma(v);
  const double Bm = dm(dm(mass, dm(gamma, gamma)), dm(v, v)) / dm(2.0, mu);
  const double X[3] = {s[1], s[2], s[3]};
  const double bp = dm(2.0 / v, fl_halfbouncepath<M>(f, s[0], X, Bm, flres, scratch + (size_t)k * stride, cap));
  const double dt = dm(bctimestep, bp);
  double* p = plan + 4 * k;
  p[0] = Bm;
  p[1] = dt;
  if (!(dt > 0.0) || !isfinite(dt)) {
    status[k] = RAPT_ST_FIELDLINE;
    if (flag) flag[k] = 1;
    p[2] = 0.0;
    return;
  }
  const double tcur = s[4];
  p[2] = ceil(da(da(tcur, delta), -tcur) / dt);  // len(np.arange(tcur, tcur + delta, dt))
  p[3] = da(da(tcur, dt), -tcur);                 // numpy's fill step for i >= 2
  status[k] = RAPT_ST_OK;
}

// Interval j of every tracer with j < K: one SciPy-dopri5 integrate() call from
// the integrator time (state t) over dt, then the row stamped with the
// interval's start, np.arange's j-th value. A team of kBcTeam lanes a tracer:
// every lane carries the same integration, and the right-hand sides are the
// team's. The loop runs until the last tracer of the warp has finished, so that
// all lanes meet in each right-hand side; a finished team repeats its last
// state (step 0). scratch: kBcLines * stride doubles a team of the launch.
template <int M>
__global__ void __launch_bounds__(64) k_bc_interval(const __grid_constant__ FieldP f, KParams P, int64_t n, double* st,
                                                    const double* cst, const double* plan, double d, int64_t j,
                                                    double* rows, int max_rows, int32_t* nrows, int32_t* status,
                                                    int64_t* counters, int32_t* flag, double* scratch,
                                                    long long stride, int cap) {
  __shared__ double gauss[16];
  if (threadIdx.x == 0) gauss_legendre8(gauss, gauss + 8);
  __syncthreads();
  const int64_t team = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kBcTeam;
  const int64_t k = team < n ? team : n - 1;
  const double* p = plan + 4 * k;
  bool live = team < n && status[k] == RAPT_ST_OK && (double)j < p[2];
  const bool writes = live && (threadIdx.x & (kBcTeam - 1)) == 0;
  if (!__any_sync(kFull, live)) return;
  double* s = st + 5 * k;
  const double v = cst[4 * k], mass = cst[4 * k + 2], charge = cst[4 * k + 3];
  const double gamma = bc_gamma(v);
  bool bad = false;
  const BcTeamRHS<M> rhs{f, p[0], dm(dm(dm(gamma, mass), v), v) / charge, d, P.flres,
                         scratch + (size_t)team * kBcLines * stride, stride, cap, gauss, &bad};
  const double dt = p[1];
  double rt = s[0];
  double y[3] = {s[1], s[2], s[3]}, k1[3];
  const double xend = da(rt, dt);
  // SciPy dopri5 (Hairer's DOPRI5, beta 0.04) over [rt, xend], restarted
  constexpr double beta = 0.04, safe = 0.9;
  constexpr double expo1 = 0.2 - beta * 0.75, facc1 = 1.0 / 0.2, facc2 = 1.0 / 10.0;
  const double hmax = fabs(xend - rt), posneg = copysign(1.0, xend - rt);
  rhs(rt, y, k1);
  double h = hinit<3>(rhs, rt, y, k1, posneg, 1.0 / 5.0, hmax, P.rtol, P.atol);
  long long nfcn = 2, nstep = 0, nacc = 0, nrej = 0;
  double facold = 1e-4;
  bool reject = false, last = false;
  int fail = 0;
  const bool ran = live;
  bool flagged = bad;
  for (;;) {
    if (live) {
      if (nstep > P.nsteps) { fail = RAPT_ST_MAXSTEPS; live = false; }
      else if (0.1 * fabs(h) <= fabs(rt) * kUround) { fail = RAPT_ST_HMIN; live = false; }
      else if ((rt + 1.01 * h - xend) * posneg > 0.0) { h = xend - rt; last = true; }
    }
    if (!__any_sync(kFull, live)) break;
    bad = false;
    double y1[3], k7[3], err;
    dopri5_attempt_rolled<3>(rhs, rt, y, k1, live ? h : 0.0, P.rtol, P.atol, y1, k7, err);
    if (live) {
      flagged = flagged || bad;
      ++nstep;
      nfcn += 6;
      const double fac11 = pow_fp64(err, expo1);
      double fac = fac11 / pow_fp64(facold, beta);
      fac = fmax(facc2, fmin(facc1, fac / safe));
      double hnew = h / fac;
      if (err <= 1.0) {
        facold = fmax(err, 1.0e-4);
        ++nacc;
        for (int i = 0; i < 3; ++i) { k1[i] = k7[i]; y[i] = y1[i]; }
        rt = rt + h;
        if (last) live = false;
        if (fabs(hnew) > hmax) hnew = posneg * hmax;
        if (reject) hnew = posneg * fmin(fabs(hnew), fabs(h));
        reject = false;
      } else {
        hnew = h / fmin(facc1, fac11 / safe);
        reject = true;
        if (nacc >= 1) ++nrej;
        last = false;
      }
      h = hnew;
    }
  }
  if (!ran || !writes) return;
  if (flagged && flag) flag[k] = 1;
  if (fail) status[k] = fail;
  if (!(isfinite(y[0]) && isfinite(y[1]) && isfinite(y[2]))) status[k] = RAPT_ST_NONFINITE;
  const double tcur0 = s[4];
  const double tj = j == 0 ? tcur0 : (j == 1 ? da(tcur0, dt) : da(tcur0, dm((double)j, p[3])));
  if (nrows[k] < max_rows) {
    double* r = rows + ((size_t)k * (size_t)max_rows + (size_t)nrows[k]) * 4;
    r[0] = tj; r[1] = y[0]; r[2] = y[1]; r[3] = y[2];
  }
  nrows[k] += 1;
  s[0] = tj;  // trajectory[-1] = (t_j, x, y, z); the integrator restarts from it
  s[1] = y[0]; s[2] = y[1]; s[3] = y[2];
  if (j + 1 >= (int64_t)p[2] || status[k] != RAPT_ST_OK) s[4] = tj;  // tcur = trajectory[-1, 0]
  if (counters) {
    int64_t* c = counters + 4 * k;
    c[0] += nfcn; c[1] += nstep; c[2] += nacc; c[3] += nrej;
  }
}

// what 0 the second invariant I, 1 grad I (3 values), 2 the drift velocity
// (3 values), 3 the half-bounce path, at tpos[n][4] with mirror fields Bm[n]
// (what 2: cst[n][4]).
template <int M>
__global__ void k_bc_eval(FieldP f, double flres, int what, int64_t n, const double* tpos, const double* Bm, double d,
                          const double* cst, double* out, double* scratch, long long stride, int cap) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double* tp = tpos + 4 * k;
  const double X[3] = {tp[1], tp[2], tp[3]};
  double* scr = scratch + (size_t)k * stride;
  double* o = out + 3 * k;
  if (what == 0 || what == 3) {
    o[0] = what == 0 ? fl_eye<M>(f, tp[0], X, Bm[k], flres, scr, cap)
                     : fl_halfbouncepath<M>(f, tp[0], X, Bm[k], flres, scr, cap);
    o[1] = o[2] = 0.0;
  } else if (what == 1) {
    fl_gradI<M>(f, tp[0], X, Bm[k], d, flres, scr, cap, o);
  } else {
    const double v = cst[4 * k], mass = cst[4 * k + 2], charge = cst[4 * k + 3];
    const double gamma = bc_gamma(v);
    const BcRHS<M> rhs{f, Bm[k], dm(dm(dm(gamma, mass), v), v) / charge, d, flres, scr, cap};
    rhs(tp[0], X, o);
  }
}

}  // namespace rapt
