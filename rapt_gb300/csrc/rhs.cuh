// rhs.cuh -- equations of motion on the device.
#pragma once
#include "fields.cuh"

namespace rapt {

// Newton-Lorentz equation, the eom closure of Particle.advance
// (rapt/Particle.py:284-298): dx/dt = p / (gamma m), dp/dt = q (E + p x B / (gamma m)).
// gamma m is frozen at the start of the advance() call when the field is
// static and recomputed from the stage momentum otherwise, as in the reference.
template <int M>
struct ParticleRHS {
  const FieldP& f;  // in the kernel's parameter space (__grid_constant__)
  double charge, mass2, inv_gm_frozen;
  bool eq;
  __device__ __forceinline__ void operator()(double t, const double* Y, double* o) const {
    double igm = inv_gm_frozen;
    if (!field_static<M>(f)) igm = rsqrt(mass2 + (Y[3] * Y[3] + Y[4] * Y[4] + Y[5] * Y[5]) * (1.0 / (kC * kC)));
    double B[3], E[3];
    field_BE<M>(f, t, Y[0], Y[1], Y[2], B, E);
    o[0] = Y[3] * igm;
    o[1] = Y[4] * igm;
    o[2] = Y[5] * igm;
    const double qg = charge * igm;
    o[3] = qg * (Y[4] * B[2] - Y[5] * B[1]);
    o[4] = qg * (Y[5] * B[0] - Y[3] * B[2]);
    o[5] = qg * (Y[3] * B[1] - Y[4] * B[0]);
    if (Field<M>::kHasE) {
      o[3] = charge * E[0] + qg * (Y[4] * B[2] - Y[5] * B[1]);
      o[4] = charge * E[1] + qg * (Y[5] * B[0] - Y[3] * B[2]);
      o[5] = charge * E[2] + qg * (Y[3] * B[1] - Y[4] * B[0]);
    }
    if (eq) { o[2] = 0.0; o[5] = 0.0; }
  }
};

// Guiding-centre equations (rapt/GuidingCenter.py:329-395).
//   eom 0: Tao-Chan-Brizard   (GuidingCenter.py:329-355)
//   eom 1: Brizard-Chan       (GuidingCenter.py:357-379)
//   eom 2: Northrop-Teller    (GuidingCenter.py:381-395)
// grad|B| and curl b use the reference's central differences with the field's
// gradientstepsize, evaluated on the 6-point stencil once (7 B evaluations per
// call for static fields instead of the reference's 13; same values).
template <int M>
struct GcRHS {
  const FieldP& f;  // in the kernel's parameter space (__grid_constant__)
  double charge, qinv, mu, minv, k_mu, inv_mc;  // k_mu = 2 mu/(m c^2), inv_mc = 1/(m c)
  double inv_gamma_v, gm_v, gm_v_v2;             // BC/NT: 1/gamma(v), gamma(v) m, gamma m v^2
  int eom;
  bool eq;
  __device__ __forceinline__ void operator()(double t, const double* Y, double* o) const {
    double ub[3], Bmag, B[3], gB[3], cb[3], E[3] = {0.0, 0.0, 0.0}, db[3] = {0.0, 0.0, 0.0};
    if constexpr (M == RAPT_GRID) {
      // B, E, the stencil and db/dt from one cell search (grid_gc_fields)
      const GridFields g = grid_gc_fields(RAPT_GRID_PASS(f), f.gB, eom == 0 ? f.gE : nullptr, t, Y[0], Y[1], Y[2],
                                          f.gradstep, f.inv2d, f.timestep, eom == 0 && !field_static<M>(f));
#pragma unroll
      for (int k = 0; k < 3; ++k) { B[k] = g.B[k]; E[k] = g.E[k]; gB[k] = g.gB[k]; cb[k] = g.cb[k]; db[k] = g.db[k]; }
      centre(B, ub, Bmag);
    } else {
      const double tm = Field<M>::time(f, t);
      stencil_sample<M>(f, tm, Y[0], Y[1], Y[2], false, B);
      centre(B, ub, Bmag);
      stencil_gradB_curlb<M>(f, tm, Y, ub, Bmag, gB, cb);
      if (eom == 0 && !Field<M>::kStatic) {
        if (Field<M>::kHasE) Field<M>::E(f, t, Y[0], Y[1], Y[2], E);
        if (Field<M>::kTimeB) {
          dbdt<M>(f, t, Y, db);
        } else {
#pragma unroll
          for (int k = 0; k < 3; ++k) db[k] = (ub[k] - ub[k]) * (0.5 / f.timestep);
        }
      }
    }
    equations(Y[3], B, ub, Bmag, gB, cb, E, db, o);
  }
  __device__ __forceinline__ static void centre(const double* B, double* ub, double& Bmag) {
    if constexpr (M != RAPT_GRID) {
      sample_unit_and_mag<M>(B, ub, Bmag);
    } else {
      const double b2 = dot3(B, B);
      const double ib = rsqrt(b2);
      Bmag = b2 * ib;
      ub[0] = B[0] * ib; ub[1] = B[1] * ib; ub[2] = B[2] * ib;
    }
  }
  // The slopes from the field at the guiding centre: B, b, |B|, grad|B|, curl b,
  // E and db/dt (the last two of the Tao-Chan-Brizard equations only).
  __device__ __forceinline__ void equations(double ppar, const double* B, const double* ub, double Bmag,
                                            const double* gB, const double* cb, const double* E, const double* db,
                                            double* o) const {
    if (eom == 0) {
      const double pm = ppar * inv_mc;
      const double g2 = 1.0 + k_mu * Bmag + pm * pm;
      const double rg = rsqrt(g2);
      const double pq = ppar * qinv;
      double Bs[3] = {B[0] + pq * cb[0], B[1] + pq * cb[1], B[2] + pq * cb[2]};
      const double iBsp = 1.0 / dot3(Bs, ub);
      const double mg = mu * rg;
      double Es[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        // the zero terms of static models and of models without E are left out
        const double g = Field<M>::kStatic ? mg * gB[i] : ppar * db[i] + mg * gB[i];
        Es[i] = Field<M>::kHasE ? E[i] - g * qinv : -(g * qinv);
      }
      double Exb[3];
      cross3(Es, ub, Exb);
      const double a = ppar * rg * minv;
#pragma unroll
      for (int i = 0; i < 3; ++i) o[i] = (a * Bs[i] + Exb[i]) * iBsp;
      o[3] = charge * dot3(Es, Bs) * iBsp;
    } else if (eom == 1) {
      const double pq = ppar * qinv;
      double Bs[3] = {B[0] + pq * cb[0], B[1] + pq * cb[1], B[2] + pq * cb[2]};
      const double iBsp = 1.0 / dot3(Bs, ub);
      double bxg[3];
      cross3(ub, gB, bxg);
      const double a = ppar * inv_gamma_v * minv;
      const double c = mu * qinv * inv_gamma_v;
#pragma unroll
      for (int i = 0; i < 3; ++i) o[i] = (a * Bs[i] + c * bxg[i]) * iBsp;
      o[3] = -mu * dot3(Bs, gB) * inv_gamma_v * iBsp;
    } else {
      double bxg[3];
      cross3(ub, gB, bxg);
      const double s = (gm_v_v2 + ppar * ppar / gm_v) / (2.0 * charge * Bmag * Bmag);
      const double a = ppar / gm_v;
#pragma unroll
      for (int i = 0; i < 3; ++i) o[i] = s * bxg[i] + a * ub[i];
      o[3] = -mu * dot3(ub, gB) * inv_gamma_v;
    }
    if (eq) { o[2] = 0.0; o[3] = 0.0; }
  }
};

// ---------------------------------------------------------------- right-hand sides by teams
// An FP64 instruction holds a sub-partition's FP64 pipe for 64 cycles whether
// one lane is active or all 32 are, and a guiding-centre right-hand side in one
// lane is 350-1,800 of them in a row (seven to nine field samples). Where few
// lanes of a warp have a tracer -- a small ensemble, the end of a launch -- the
// idle lanes take the samples: a team of kTeam lanes evaluates one tracer's
// samples side by side, exchanges the differences by shuffles and forms the
// equations, ~130 instructions (Grid: ~400) for 32 / kTeam tracers at once. The
// samples and their differences are the ones operator() forms, so a tracer's
// result does not depend on which lanes worked on it. Per advance, one tracer a
// lane only -> with teams: one electron, 1 s in the double dipole 18.1 -> 8.1 ms;
// 10,007 with dense rows 14.9 -> 11.0 ms; 65,536 over 0.5 s (the end of the
// launch) 37.8 -> 34.8 ms; 16,384 in a 121^3 grid 213 -> 84 ms.
template <int M>
struct GcTeam {
  static constexpr bool kTimed = Field<M>::kTimeB;              // samples 7 and 8: t -+ ts
  static constexpr int kTeam = kTimed ? 16 : 8;
  static constexpr int kTeams = 32 / kTeam;
  // rounds of a team against one right-hand side a lane: the largest number of
  // busy lanes for which the teams take less of the pipe
  static constexpr int kMaxLanes = kTimed ? (M == RAPT_GRID ? 8 : 6) : (M == RAPT_HARRIS ? 4 : 12);
};

__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(kFull, v, src); }

struct Quad {
  double v0, v1, v2, v3;
};
// Per-tracer constants of the guiding-centre equations (GcRHS).
struct GcConst {
  double charge, qinv, mu, minv, k_mu, inv_mc, inv_gamma_v, gm_v, gm_v_v2;
};

// Right-hand sides at (t, Y) for the lanes of the mask `left`, by teams; called
// by all 32 lanes. Sample j of a team: 2a, 2a + 1 at x +- d e_a, 6 the centre,
// 7 and 8 at t -+ ts, 9 E of a Grid.
template <int M>
static __device__ __noinline__ Quad gc_rhs_teams(unsigned left, const FieldP& f, int eom, bool eq, double t, Quad Yv,
                                                 GcConst c) {
  using G = GcTeam<M>;
  const int lane = threadIdx.x & 31, j = lane & (G::kTeam - 1), team = lane / G::kTeam, base = lane - j;
  Quad out{0.0, 0.0, 0.0, 0.0};
  while (left) {
    // the team's tracer: the team-th of the lanes left (the first for a team without one)
    const int busy = __popc(left);
    unsigned rest = left;
#pragma unroll
    for (int k = 0; k < G::kTeams - 1; ++k)
      if (team < busy && k < team) rest &= rest - 1u;
    const int src = __ffs(rest) - 1;
    const double tt = shfl_d(t, src);
    const double y[4] = {shfl_d(Yv.v0, src), shfl_d(Yv.v1, src), shfl_d(Yv.v2, src), shfl_d(Yv.v3, src)};
    const GcRHS<M> r{f, shfl_d(c.charge, src), shfl_d(c.qinv, src), shfl_d(c.mu, src), shfl_d(c.minv, src),
                     shfl_d(c.k_mu, src), shfl_d(c.inv_mc, src), shfl_d(c.inv_gamma_v, src), shfl_d(c.gm_v, src),
                     shfl_d(c.gm_v_v2, src), eom, eq};
    // this lane's sample
    const double d = (j & 1) ? -f.gradstep : f.gradstep;
    const int axis = j < 6 ? j >> 1 : 3;
    const double x0 = axis == 0 ? y[0] + d : y[0], x1 = axis == 1 ? y[1] + d : y[1], x2 = axis == 2 ? y[2] + d : y[2];
    double ts = tt;
    if (G::kTimed) ts = j == 7 ? tt - f.timestep : (j == 8 ? tt + f.timestep : tt);
    double b[3], u[3], m;
    if constexpr (M == RAPT_GRID) {
      const bool es = j == 9 && f.gE;
      const GridV v = grid_interp(RAPT_GRID_PASS(f), es ? f.gE : f.gB, ts, x0, x1, x2);
      b[0] = v.a; b[1] = v.b; b[2] = v.c;
    } else {
      stencil_sample<M>(f, Field<M>::time(f, ts), x0, x1, x2, axis == 2, b);
    }
    sample_unit_and_mag<M>(b, u, m);
    // the centre's sample, and the differences of each pair to every lane
    const double B[3] = {shfl_d(b[0], base + 6), shfl_d(b[1], base + 6), shfl_d(b[2], base + 6)};
    const double ub[3] = {shfl_d(u[0], base + 6), shfl_d(u[1], base + 6), shfl_d(u[2], base + 6)};
    const double Bmag = shfl_d(m, base + 6);
    double du[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) du[i] = u[i] - __shfl_xor_sync(kFull, u[i], 1);
    const double dmag = m - __shfl_xor_sync(kFull, m, 1);
    const double gB[3] = {shfl_d(dmag, base) * f.inv2d, shfl_d(dmag, base + 2) * f.inv2d,
                          shfl_d(dmag, base + 4) * f.inv2d};
    const double c0 = shfl_d(du[2], base + 2) - shfl_d(du[1], base + 4);
    const double c1 = shfl_d(du[0], base + 4) - shfl_d(du[2], base);
    const double c2 = shfl_d(du[1], base) - shfl_d(du[0], base + 2);
    const double cb[3] = {c0 * f.inv2d, c1 * f.inv2d, c2 * f.inv2d};
    double E[3] = {0.0, 0.0, 0.0}, db[3] = {0.0, 0.0, 0.0};
    if (!Field<M>::kStatic && eom == 0) {
      if (M == RAPT_GRID) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double e = shfl_d(b[i], base + 9);
          if (f.gE) E[i] = e;
        }
      } else if (Field<M>::kHasE) {
        Field<M>::E(f, tt, y[0], y[1], y[2], E);
      }
      if (!field_static<M>(f)) {
        const double h = 0.5 / f.timestep;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          db[i] = (G::kTimed ? shfl_d(u[i], base + 8) - shfl_d(u[i], base + 7) : ub[i] - ub[i]) * h;
      }
    }
    double o[4];
    r.equations(y[3], B, ub, Bmag, gB, cb, E, db, o);
    // back to the lanes served in this round
    const int rank = __popc(left & ((1u << lane) - 1u));
    const bool mine = (left >> lane & 1u) && rank < G::kTeams;
    const int from = (mine ? rank : 0) * G::kTeam;
    const Quad v{shfl_d(o[0], from), shfl_d(o[1], from), shfl_d(o[2], from), shfl_d(o[3], from)};
    if (mine) out = v;
#pragma unroll
    for (int k = 0; k < G::kTeams; ++k) left &= left - 1u;  // 0 stays 0
  }
  return out;
}

// The right-hand side of the lanes with `need` set as a functor that all 32
// lanes of a warp call together: a lane's own, or the teams' where few lanes
// need one. The other lanes' o is left as it was.
template <int M>
struct GcWarpRHS {
  const GcRHS<M>& r;
  bool need;
  __device__ __forceinline__ void operator()(double t, const double* Y, double* o) const {
    const unsigned left = __ballot_sync(kFull, need);
    if (__popc(left) > GcTeam<M>::kMaxLanes) {
      if (need) r(t, Y, o);
    } else {
      const Quad v = gc_rhs_teams<M>(left, r.f, r.eom, r.eq, t, Quad{Y[0], Y[1], Y[2], Y[3]},
                                     GcConst{r.charge, r.qinv, r.mu, r.minv, r.k_mu, r.inv_mc, r.inv_gamma_v, r.gm_v,
                                             r.gm_v_v2});
      if (need) { o[0] = v.v0; o[1] = v.v1; o[2] = v.v2; o[3] = v.v3; }
    }
  }
};

}  // namespace rapt
