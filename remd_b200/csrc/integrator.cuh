// integrator.cuh -- the Nose-Poincare thermostat / Andersen barostat quaternion
// integrator of the reference (src/integrator.cxx:132-706), FP64, split into
// the per-replica scalar chain (run by one thread and broadcast) and the
// per-molecule free-rotor / drift / kick operators (one thread per molecule).
//
// Operation order follows the reference CPU code so the FP64 results agree
// with it to rounding; confined=2 (slit) barostat terms follow the reference
// GPU kernel (src/remdgpu.cu:2083-2120, 2537-2545, 2803-2809), since the
// reference CPU slit path does not run (src/force_calculator.cxx:1525, 1556-1561).
#pragma once
#include "engine_types.cuh"

namespace remd {

__host__ __device__ inline double volume(const RepConst& c, const RepState& st) {
  // Molecules::GetVolume / GetBottomArea, src/molecules.h:357-376
  if (c.confined == 1) return c.bottom_area * st.L[2];
  if (c.confined == 2) return st.L[0] * st.L[1] * c.slit_width;
  return st.L[0] * st.L[1] * st.L[2];
}

// D6: thermostat half step, src/integrator.cxx:634-644
__device__ inline void d6(const RepConst& c, RepState& st) {
  if (c.tconstant == 1) {
    const double tmp = 1.0 + st.Ps * c.hQ;   // hQ = (dt/2) / (2 Q)
    st.s *= tmp * tmp;
    st.Ps /= tmp;
  }
}

// D5 scalar part (src/integrator.cxx:583-600; slit src/remdgpu.cu:2537-2545), in two:
// the terms that depend on the forces and the box only (the closing and the opening
// D5 of a step share them), and their use.
struct D5Terms {
  double Ps, Pv[3];   // added to Ps, and, times s, to Pv
};
__device__ inline D5Terms d5_terms(const RepConst& c, const RepState& st, double pot, const double* vir) {
  const double h = c.dthalf;
  D5Terms t = {0.0, {0.0, 0.0, 0.0}};
  if (c.tconstant == 1) t.Ps = -(c.pconstant > 0 ? pot + st.P * volume(c, st) : pot) * h;
  if (c.pconstant == 1)
    t.Pv[0] = ((vir[0] + vir[1] + vir[2]) / (3.0 * st.L[0] * st.L[1] * st.L[2]) - st.P) * h;
  if (c.pconstant == 2) t.Pv[2] = (vir[2] / st.L[2] - st.P * c.bottom_area) * h;
  if (c.pconstant == 3) {
    const double zlen = (c.confined == 2) ? c.wall_length_param : st.L[2];
    t.Pv[0] = (vir[0] / st.L[0] - st.P * st.L[1] * zlen) * h;
    t.Pv[1] = (vir[1] / st.L[1] - st.P * st.L[0] * zlen) * h;
  }
  return t;
}
__device__ inline void d5_apply(RepState& st, const D5Terms& t) {
  st.Ps += t.Ps;
  for (int x = 0; x < 3; x++) st.Pv[x] += st.s * t.Pv[x];
}

// x^(1/3) as the reference takes it, powf(float, float) with the float 1/3
// (src/integrator.cxx:614), evaluated in double and rounded once to float, i.e. the
// correctly rounded single-precision result: x^(1/3 + e) = cbrt(x) (1 + e ln x),
// e = (float)(1/3) - 1/3 = 1e-8; the neglected (e ln x)^2 / 2 and the single-precision
// logarithm are below 1e-13 relative.
__device__ inline double box_cbrt(float x) {
  const double e = (double)(1.f / 3.f) - 1.0 / 3.0;
  return (double)(float)(cbrt((double)x) * (1.0 + e * (double)logf(x)));
}

// D4: barostat half step, src/integrator.cxx:604-632 (slit: src/remdgpu.cu:2096-2115)
__device__ inline void d4(const RepConst& c, RepState& st) {
  const double dthalf = c.dthalf;
  if (c.pconstant == 1) {
    if (c.tconstant == 1) st.Ps -= st.Pv[0] * st.Pv[0] * c.iW * dthalf;
    st.L[0] = st.L[1] = st.L[2] = box_cbrt((float)(volume(c, st) + st.Pv[0] * st.s * c.iW * dthalf));
  }
  if (c.pconstant == 2) {
    if (c.tconstant == 1) st.Ps -= 0.5 * st.Pv[2] * st.Pv[2] * c.iW * dthalf;
    st.L[2] += st.s * st.Pv[2] * c.iW * dthalf;
  }
  if (c.pconstant == 3) {
    const double bw = 0.5 * c.iW;
    if (c.tconstant == 1) st.Ps -= (st.Pv[0] * st.Pv[0] + st.Pv[1] * st.Pv[1]) * bw * dthalf;
    st.L[0] += st.s * st.Pv[0] * bw * c.dt;
    st.L[1] += st.s * st.Pv[1] * bw * c.dt;
  }
}

// D3D2D1D2D3_PsPv, src/integrator.cxx:132-172; log_s = log(st.s)
__device__ inline void pspv(const RepConst& c, RepState& st, const double* sum_Pv, double sum_Ps, double log_s) {
  double k[3] = {0.0, 0.0, 0.0};
  if (c.pconstant > 0 || c.tconstant == 1)
    for (int d = 0; d < 3; d++) k[d] = sum_Pv[d] / (st.L[d] * st.L[d] * st.s * st.s);
  const double sPv = k[0] + k[1] + k[2];
  if (c.pconstant == 1) st.Pv[0] += st.s * sPv / (volume(c, st) * 3.0) * c.dthalf;
  if (c.pconstant == 2) st.Pv[2] += st.s * k[2] / st.L[2] * c.dthalf;
  if (c.pconstant == 3) {
    st.Pv[0] += st.s * k[0] / st.L[0] * c.dthalf;
    st.Pv[1] += st.s * k[1] / st.L[1] * c.dthalf;
  }
  if (c.tconstant == 1) st.Ps += (0.25 * sPv + 2.0 * sum_Ps - (1.0 + log_s) * st.gkT + st.H0) * c.dt;
}

// body_to_space / space_to_body, src/rotation.h:146-187
__host__ __device__ inline void body_to_space(const double* a, const double* v, double* o) {
  const double a0sq = a[0] * a[0], a1sq = a[1] * a[1], a2sq = a[2] * a[2], a3sq = a[3] * a[3];
  const double a01 = a[0] * a[1], a02 = a[0] * a[2], a03 = a[0] * a[3];
  const double a12 = a[1] * a[2], a13 = a[1] * a[3], a23 = a[2] * a[3];
  o[0] = (a0sq + a1sq - a2sq - a3sq) * v[0] + 2. * (a12 - a03) * v[1] + 2. * (a13 + a02) * v[2];
  o[1] = 2. * (a12 + a03) * v[0] + (a0sq - a1sq + a2sq - a3sq) * v[1] + 2. * (a23 - a01) * v[2];
  o[2] = 2. * (a13 - a02) * v[0] + 2. * (a23 + a01) * v[1] + (a0sq - a1sq - a2sq + a3sq) * v[2];
}

__host__ __device__ inline void space_to_body(const double* a, const double* v, double* o) {
  const double a0sq = a[0] * a[0], a1sq = a[1] * a[1], a2sq = a[2] * a[2], a3sq = a[3] * a[3];
  const double a01 = a[0] * a[1], a02 = a[0] * a[2], a03 = a[0] * a[3];
  const double a12 = a[1] * a[2], a13 = a[1] * a[3], a23 = a[2] * a[3];
  o[0] = (a0sq + a1sq - a2sq - a3sq) * v[0] + 2. * (a12 + a03) * v[1] + 2. * (a13 - a02) * v[2];
  o[1] = 2. * (a12 - a03) * v[0] + (a0sq - a1sq + a2sq - a3sq) * v[1] + 2. * (a23 + a01) * v[2];
  o[2] = 2. * (a13 + a02) * v[0] + 2. * (a23 - a01) * v[1] + (a0sq - a1sq - a2sq + a3sq) * v[2];
}

// sin and cos: their Taylor polynomials to x^13 and x^14 for |x| <= 1/4 (the next
// terms are below 1e-21), where every rotation of a step falls (xi dt is a few
// hundredths); sincos beyond.  Shorter dependent chains than sincos: the integrate
// kernel is bound by FP64 latency.
__device__ inline void sincos_small(double x, double* sn, double* cs) {
  if (fabs(x) <= 0.25) {
    const double y = x * x, y2 = y * y, y4 = y2 * y2;
    const double s0 = fma(y, 1.0 / 120.0, -1.0 / 6.0), s1 = fma(y, 1.0 / 362880.0, -1.0 / 5040.0),
                 s2 = fma(y, 1.0 / 6227020800.0, -1.0 / 39916800.0);
    const double c0 = fma(y, 1.0 / 24.0, -0.5), c1 = fma(y, 1.0 / 40320.0, -1.0 / 720.0),
                 c2 = fma(y, 1.0 / 479001600.0, -1.0 / 3628800.0);
    const double c3 = -1.0 / 87178291200.0;
    *sn = fma(x * y, fma(y4, s2, fma(y2, s1, s0)), x);
    *cs = fma(y, fma(y4, fma(y2, c3, c2), fma(y2, c1, c0)), 1.0);
  } else {
    sincos(x, sn, cs);
  }
}

// The free-rotor sub-step about body axis `axis` (D1: x, D2: y, D3: z),
// src/integrator.cxx:467-563: (q,p) -> (q cos + P_k(q) sin, p cos + P_k(p) sin).
__device__ inline double rotate(double* q, double* p, int axis, double iIk, double coef_xi, double h) {
  double Pq[4], Pp[4];
  if (axis == 1) {
    Pq[0] = -q[1]; Pq[1] = q[0]; Pq[2] = q[3]; Pq[3] = -q[2];
    Pp[0] = -p[1]; Pp[1] = p[0]; Pp[2] = p[3]; Pp[3] = -p[2];
  } else if (axis == 2) {
    Pq[0] = -q[2]; Pq[1] = -q[3]; Pq[2] = q[0]; Pq[3] = q[1];
    Pp[0] = -p[2]; Pp[1] = -p[3]; Pp[2] = p[0]; Pp[3] = p[1];
  } else {
    Pq[0] = -q[3]; Pq[1] = q[2]; Pq[2] = -q[1]; Pq[3] = q[0];
    Pp[0] = -p[3]; Pp[1] = p[2]; Pp[2] = -p[1]; Pp[3] = p[0];
  }
  const double xi = (((p[0] * Pq[0] + p[1] * Pq[1]) + p[2] * Pq[2]) + p[3] * Pq[3]) * (coef_xi * iIk);
  double sn, cs;
  sincos_small(xi * h, &sn, &cs);
  for (int k = 0; k < 4; k++) q[k] = q[k] * cs + Pq[k] * sn;
  for (int k = 0; k < 4; k++) p[k] = p[k] * cs + Pp[k] * sn;
  return xi;
}

// D5 per-molecule kick (src/integrator.cxx:572-582): v += f*coef_v, p += S(q) n coef_p; coef_v = L s (dt/2) / m
__device__ inline void kick(double* v, double* p, const double* q, const double* f, const double* n,
                            const double* coef_v, double coef_p) {
  for (int d = 0; d < 3; d++) v[d] += f[d] * coef_v[d];
  const double Sn0 = ((q[0] * n[0] + (-q[1]) * n[1]) + (-q[2]) * n[2]) + (-q[3]) * n[3];
  const double Sn1 = ((q[1] * n[0] + q[0] * n[1]) + (-q[3]) * n[2]) + q[2] * n[3];
  const double Sn2 = ((q[2] * n[0] + q[3] * n[1]) + q[0] * n[2]) + (-q[1]) * n[3];
  const double Sn3 = ((q[3] * n[0] + (-q[2]) * n[1]) + q[1] * n[2]) + q[0] * n[3];
  p[0] += Sn0 * coef_p;
  p[1] += Sn1 * coef_p;
  p[2] += Sn2 * coef_p;
  p[3] += Sn3 * coef_p;
}

// Per-molecule kinetic terms of CalcProperties (src/molecules.cxx:631-657):
// tra3 += (v*v)*m per dimension; rot += I*xi*xi*2 with xi = p.P_k(q) * (1/I)*coef.
__device__ inline double rot_energy(const double* q, const double* p, const double* I, double s) {
  const double coef = 0.25 / s;
  double xi[3];
  xi[0] = ((p[0] * (-q[1]) + p[1] * q[0]) + p[2] * q[3]) + p[3] * (-q[2]);
  xi[1] = ((p[0] * (-q[2]) + p[1] * (-q[3])) + p[2] * q[0]) + p[3] * q[1];
  xi[2] = ((p[0] * (-q[3]) + p[1] * q[2]) + p[2] * (-q[1])) + p[3] * q[0];
  double r = 0.0;
  for (int k = 0; k < 3; k++) {
    const double x = xi[k] * ((1.0 / I[k]) * coef);
    r += I[k] * x * x * 2.0;
  }
  return r;
}

}  // namespace remd
