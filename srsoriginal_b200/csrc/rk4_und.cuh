// RK4 steps through ideal undulators along z without taper, the common case of a trajectory (rk4_lanes.cu,
// rk4_exact.cu; compiled with -fmad=false).  The operations and their order are field_one's, force's and
// the serial kernel's (rk4_fields.cuh, rk4.cu), so the results are theirs bit for bit; what is left out is
// exact: products with the direction's zeros and one, the taper's 1 + 0 D, sums with zero.  Only the
// stages' z is formed, and the sines of two stages run side by side: their phases are below 1e5 for every state of
// a trajectory (undulators_along_z bounds them), which lets the compiler drop sin's large-argument branch and
// interleave two calls (two calls 533 -> 356 cycles).  A caller whose states are only iterates keeps them within that
// bound.
#pragma once

#include <cuda_runtime.h>

#include "rk4_fields.cuh"

namespace srs {
namespace {

constexpr int kMaxUndulators = 2;

struct UndField {
  double Cz, ps, plen, rplen;
  double edge[6];  // region bounds in D = z - Cz, ascending: field 0 | 1/4 | 3/4 | 1 | 3/4 | 1/4 | 0
  double F[3];
};

__device__ inline void prepare_undulator(const srs_field &f, UndField &u) {
  Prepared p;
  prepare(f, p);
  u.Cz = p.C[2];
  u.ps = p.ps;
  u.plen = p.plen;
  u.rplen = p.rplen;
  u.edge[0] = p.b_lo; u.edge[1] = p.e2_lo; u.edge[2] = p.e1_lo;
  u.edge[3] = p.e1_hi; u.edge[4] = p.e2_hi; u.edge[5] = p.b_hi;
  for (int c = 0; c < 3; ++c) u.F[c] = p.F[c];
}

__device__ __forceinline__ double und_phase(const UndField &f, double D) {
  return div_rn(two_pi() * (D - f.ps), f.plen, f.rplen);
}

// field_one's value at D for the sine s, added to the field sum's zero as field_sum starts it: a component of -0
// (a field component of zero, or outside) is +0, as there; the fused operation rounds the product as a multiplication
// does.
__device__ __forceinline__ V3 und_value(const UndField &f, double D, double s) {
  const double *e = f.edge;
  const bool out = D > e[5] || D < e[0], end = D < e[2] || D > e[3], tip = D < e[1] || D > e[4];
  const double fac = out ? 0.0 : end ? (tip ? 0.25 : 0.75) : 1.0;
  return v3(__fma_rn(f.F[0] * fac, s, 0.0), __fma_rn(f.F[1] * fac, s, 0.0), __fma_rn(f.F[2] * fac, s, 0.0));
}

__device__ __forceinline__ double und_sine(double x) {
  __builtin_assume(fabs(x) < 1.0e5);
  __builtin_assume(x == x);
  return sin(x);
}

// The field at two heights za and zb
template <int kN>
__device__ __forceinline__ void und_fields(const UndField *f, double za, double zb, V3 &Ba, V3 &Bb) {
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    const double Da = za - f[i].Cz, Db = zb - f[i].Cz;
    const double sa = und_sine(und_phase(f[i], Da)), sb = und_sine(und_phase(f[i], Db));
    const V3 a = und_value(f[i], Da, sa), b = und_value(f[i], Db, sb);
    Ba = i == 0 ? a : Ba + a;
    Bb = i == 0 ? b : Bb + b;
  }
}

// The quantities of one RK4 step that depend on the state only weakly: r1 = hh*a1, r2 = hh*a2, r3 = h*a3,
// d = h6*(a1 + a4 + 2(a3 + a2)).
struct Increments {
  V3 r1, r2, r3, d, a1;
};

__device__ __forceinline__ V3 scale3(double s, V3 a) { return v3(s * a.x, s * a.y, s * a.z); }

template <int kN>
__device__ __forceinline__ Increments und_increments(const UndField *f, double qomg, double h, double hh, double h6,
                                                     V3 pos, V3 vel) {
  Increments o;
  V3 B1, B2, B3, B4;
  und_fields<kN>(f, pos.z, pos.z + hh * vel.z, B1, B2);
  o.a1 = force(qomg, vel, B1);
  o.r1 = scale3(hh, o.a1);
  const V3 v2 = vel + o.r1;
  const V3 a2 = force(qomg, v2, B2);
  o.r2 = scale3(hh, a2);
  const V3 v3_ = vel + o.r2;
  und_fields<kN>(f, pos.z + hh * v2.z, pos.z + h * v3_.z, B3, B4);
  const V3 a3 = force(qomg, v3_, B3);
  o.r3 = scale3(h, a3);
  const V3 v4 = vel + o.r3;
  const V3 a4 = force(qomg, v4, B4);
  const V3 m = a3 + a2;
  o.d = v3(h6 * (o.a1.x + a4.x + 2.0 * m.x), h6 * (o.a1.y + a4.y + 2.0 * m.y), h6 * (o.a1.z + a4.z + 2.0 * m.z));
  return o;
}

// the position increment of a component: h6*((v + v4) + 2(v3 + v2))
__device__ __forceinline__ double advance(double h6, double v, double r1, double r2, double r3) {
  const double v2 = v + r1, v3_ = v + r2, v4 = v + r3;
  return h6 * (v + v4 + 2.0 * (v3_ + v2));
}

}  // namespace
}  // namespace srs
