// Hand-written adjoint (reverse-mode derivative) of the on-axis spectrum and of the RK4 trajectory.
//
// The forward path is: initial state s0 = (x0, v0) and the fields -> RK4 states s_j (stored as the
// trajectory points x_j, beta_j = v_j / c) -> the sums E_k = Sum_i f_i(w_k) -> flux_k = C2 (C0 w_k dt)^2
// |E_k|^2 (OSCARSSR.cc:1154-1251).  Given dL/dflux_k this file computes dL/d(field parameters),
// dL/dx0, dL/dbeta0 and dL/d(q/(m gamma)).
//
// 1. Sum adjoint (spectrum_adjoint_kernel): four lanes per trajectory point i, looping over the
//    energies, give g_i = dL/d(x_i, beta_i) in closed form (derivatives of the amplitude
//    (beta - n(1 + i c/(w D)))/D and of the phase w (i dt + D/c) with respect to x and beta).
// 2. Trajectory adjoint: lambda_j = dL/ds_j obeys lambda_j = g_j + J_j^T lambda_{j+1}, where J_j is
//    the Jacobian of RK4 step j.  Instead of one serial sweep back through the N steps (the forward
//    RK4 is a serial chain; its adjoint need not be), the affine recurrence is solved as a scan:
//      (a) every step's 6 x 6 Jacobian is formed in parallel from the stored states, by forward-mode
//          tangents pushed through the four stages, and chunks of kAdjChunk steps are composed there into affine maps
//          lambda_j0 = M lambda_j1 + b (step_maps_kernel);
//      (b) one warp carries lambda across the chunk maps from the last point back to the first
//          (carry_kernel);
//      (c) each chunk carries its end value across its steps with the stored Jacobians; then all steps run
//          the reverse-mode step from their own lambda at once
//          (VJP through the four stages, recomputed from the stored state), which yields the
//          field-parameter and q/(m gamma) contributions (finish_kernel).
//    The stored trajectory is itself the checkpoint set: the state at every step is in HBM (the sums
//    need every point anyway), so each step's stages are recomputed from its own stored state and
//    no sqrt(N) re-integration is needed.  The reverse pass does not re-run the forward integration.
// Both chains of the reference's trajectory are handled: forward from t0 with +dt (points nbwd ..
// n-1) and backward with -dt (points nbwd-1 .. 0), both starting from s0.
//
// States are in (x [m], beta) units so that the Jacobian entries are of comparable size.  All
// arithmetic is FP64.  Grid-sample gradients are accumulated with FP64 atomics (sub-ulp
// run-to-run differences); everything else is reduced in a fixed order.
#include <cuda_runtime.h>

#include <cuda_pipeline.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "srs_device.cuh"
#include "srs_internal.h"

namespace srs {
namespace {

constexpr int kAdjChunk = 16;     // steps per scan chunk
constexpr int kAdjBlock = 128;    // steps (and threads) per block
constexpr int kAdjChunks = kAdjBlock / kAdjChunk;
constexpr int kAdjMaxFields = 16;

__device__ inline void rot_matrix(const double r[3], double R[3][3]) {
  // R[i][j] = component i of rotate_xyz(e_j): the linear map the reference applies to the point
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    V3 e = v3(j == 0, j == 1, j == 2);
    rotate_xyz(e, r);
    R[0][j] = e.x;
    R[1][j] = e.y;
    R[2][j] = e.z;
  }
}
__device__ inline bool has_rotation(const double r[3]) { return r[0] != 0 || r[1] != 0 || r[2] != 0; }

// Corners of the grid interpolation at X: sample indices, weights and d(weight)/dX' per axis, where
// X' = R X - translation is the point in the grid's frame (TField3D_Grid.cc:124-243).  nc = 0 outside.
struct Corners {
  int nc;
  int64_t idx[8];
  double w[8];
  double dw[8][3];
};

__device__ void grid_corners(const srs_field &f, V3 XIN, Corners &C) {
  V3 X = XIN;
  if (has_rotation(f.rotations)) rotate_xyz(X, f.rotations);
  X = X - ld3(f.translation);
  const double xs[3] = {X.x, X.y, X.z};
  bool act[3];
  int64_t base[3];
  double t[3];
  C.nc = 0;
  for (int a = 0; a < 3; ++a) {
    act[a] = f.n[a] > 1;
    base[a] = 0;
    t[a] = 0;
    if (!act[a]) continue;
    if (xs[a] <= f.start[a] || xs[a] >= f.start[a] + (double)(f.n[a] - 1) * f.step[a]) return;
    uint64_t k = (uint64_t)((xs[a] - f.start[a]) / f.step[a]);
    if (k > (uint64_t)(f.n[a] - 2)) k = f.n[a] - 2;
    base[a] = (int64_t)k;
    t[a] = ((xs[a] - f.start[a]) - (double)k * f.step[a]) / f.step[a];
  }
  int na = 0, axes[3];
  for (int a = 0; a < 3; ++a)
    if (act[a]) axes[na++] = a;
  if (na == 0) return;
  C.nc = 1 << na;
  for (int c = 0; c < C.nc; ++c) {
    int64_t id[3] = {base[0], base[1], base[2]};
    double w = 1.0;
    double dwf[3] = {1.0, 1.0, 1.0};
    for (int q = 0; q < na; ++q) {
      const int a = axes[q];
      const int bit = (c >> q) & 1;
      id[a] += bit;
      const double fa = bit ? t[a] : 1.0 - t[a];
      const double da = (bit ? 1.0 : -1.0) / f.step[a];
      for (int r = 0; r < na; ++r) dwf[axes[r]] *= (r == q) ? da : fa;
      w *= fa;
    }
    C.idx[c] = id[0] * f.n[1] * f.n[2] + id[1] * f.n[2] + id[2];
    C.w[c] = w;
    for (int a = 0; a < 3; ++a) C.dw[c][a] = act[a] ? dwf[a] : 0.0;
  }
}

// The same for a map along one axis without rotation, the usual one: cell k, the weights of its two samples and
// the weights' derivatives, as grid_corners forms them, in registers (with its corners in local memory the maps
// and finish kernels took 38 and 51 us for 20001 points, so 28 and 33).
struct AxisCorners {
  int axis;  // -1: not such a map
  bool inside;
  int64_t k;
  double w[2], dw[2];
};
__device__ __forceinline__ AxisCorners axis_corners(const srs_field &f, V3 X) {
  AxisCorners C;
  C.axis = -1;
  C.inside = false;
  if (has_rotation(f.rotations)) return C;
  if (f.n[0] == 1 && f.n[1] == 1 && f.n[2] > 1) C.axis = 2;
  else if (f.n[0] == 1 && f.n[1] > 1 && f.n[2] == 1) C.axis = 1;
  else if (f.n[0] > 1 && f.n[1] == 1 && f.n[2] == 1) C.axis = 0;
  else return C;
  const int a = C.axis;
  const double x = (a == 0 ? X.x : a == 1 ? X.y : X.z) - f.translation[a], start = f.start[a], step = f.step[a];
  const int64_t n = f.n[a];
  if (x <= start || x >= start + (double)(n - 1) * step) return C;
  uint64_t k = (uint64_t)((x - start) / step);
  if (k > (uint64_t)(n - 2)) k = n - 2;
  const double t = ((x - start) - (double)k * step) / step;
  C.inside = true;
  C.k = (int64_t)k;
  C.w[0] = 1.0 - t;
  C.w[1] = t;
  C.dw[0] = -1.0 / step;
  C.dw[1] = 1.0 / step;
  return C;
}

// Scalar profile of an amplitude field (B = field * shape) and its gradient in X.
__device__ double amp_shape(const srs_field &f, V3 X, V3 &grad) {
  grad = v3(0, 0, 0);
  if (f.kind == SRS_FIELD_UNDULATOR) {  // TField3D_IdealUndulator.cc:106-139
    const V3 per = ld3(f.period);
    const double plen = mag(per);
    const V3 u = unit(per);
    const double L = plen * (f.nperiods + 2);
    const double D = dot(X - ld3(f.center), u);
    const double ps = f.phase * plen / two_pi();
    if (D > L / 2. + ps || D < -L / 2. + ps) return 0.0;
    double a = 1.0;
    if (D < -L / 2. + ps + plen || D > L / 2. + ps - plen)
      a = (D < -L / 2. + ps + plen / 2. || D > L / 2. + ps - plen / 2.) ? 0.25 : 0.75;
    double s, c;
    sincos(two_pi() * (D - ps) / plen, &s, &c);
    const double tap = 1 + D * f.taper;
    const double dD = a * (c * (two_pi() / plen) * tap + s * f.taper);
    grad = u * dD;
    return a * s * tap;
  }
  if (f.kind == SRS_FIELD_GAUSSIAN) {  // TField3D_Gaussian.cc:88-113
    V3 xb = X;
    rotate_xyz(xb, f.rotations);
    const V3 rx = xb - ld3(f.center);
    const double r[3] = {rx.x, rx.y, rx.z};
    double frac = 1.0, g[3] = {0, 0, 0};
    for (int a = 0; a < 3; ++a)
      if (f.sigma_or_width[a] > 0) {
        const double tt = r[a] / f.sigma_or_width[a];
        frac *= exp(-(tt * tt) / 2.);
      }
    for (int a = 0; a < 3; ++a)
      if (f.sigma_or_width[a] > 0) g[a] = -frac * r[a] / (f.sigma_or_width[a] * f.sigma_or_width[a]);
    double R[3][3];
    rot_matrix(f.rotations, R);
    grad = v3(R[0][0] * g[0] + R[1][0] * g[1] + R[2][0] * g[2], R[0][1] * g[0] + R[1][1] * g[1] + R[2][1] * g[2],
              R[0][2] * g[0] + R[1][2] * g[1] + R[2][2] * g[2]);
    return frac;
  }
  if (f.kind == SRS_FIELD_UNIFORM_BOX) {  // TField3D_UniformBox.cc:93-111 (flat inside: no X gradient)
    V3 xb = X;
    rotate_xyz(xb, f.rotations);
    const V3 rx = xb - ld3(f.center);
    const double r[3] = {rx.x, rx.y, rx.z};
    for (int a = 0; a < 3; ++a)
      if (f.sigma_or_width[a] > 0 && fabs(r[a]) > fabs(f.sigma_or_width[a] / 2.)) return 0.0;
    return 1.0;
  }
  return 0.0;
}

// Sum of the fields at X and its Jacobian J[i][j] = dB_i / dX_j.
__device__ void field_jet(const srs_field *F, int nf, V3 X, V3 &B, double J[3][3]) {
  B = v3(0, 0, 0);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) J[i][j] = 0.0;
  for (int q = 0; q < nf; ++q) {
    const srs_field &f = F[q];
    if (f.kind == SRS_FIELD_GRID) {
      const AxisCorners one = axis_corners(f, X);
      if (one.axis >= 0) {
        if (!one.inside) continue;
        const V3 lo = ld3(f.data + 3 * one.k), hi = ld3(f.data + 3 * one.k + 3);
        B = B + lo * one.w[0];
        B = B + hi * one.w[1];
        const double g[3] = {lo.x * one.dw[0] + hi.x * one.dw[1], lo.y * one.dw[0] + hi.y * one.dw[1],
                             lo.z * one.dw[0] + hi.z * one.dw[1]};
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            if (j == one.axis) J[i][j] += g[i];
        continue;
      }
      Corners C;
      grid_corners(f, X, C);
      if (C.nc == 0) continue;
      double dBp[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};  // dB/dX' (grid frame)
      for (int c = 0; c < C.nc; ++c) {
        const V3 s = ld3(f.data + 3 * C.idx[c]);
        B = B + s * C.w[c];
        for (int a = 0; a < 3; ++a) {
          dBp[0][a] += s.x * C.dw[c][a];
          dBp[1][a] += s.y * C.dw[c][a];
          dBp[2][a] += s.z * C.dw[c][a];
        }
      }
      if (has_rotation(f.rotations)) {
        double R[3][3];
        rot_matrix(f.rotations, R);
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) J[i][j] += dBp[i][0] * R[0][j] + dBp[i][1] * R[1][j] + dBp[i][2] * R[2][j];
      } else {
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) J[i][j] += dBp[i][j];
      }
    } else {
      V3 g;
      const double sh = amp_shape(f, X, g);
      const V3 A = ld3(f.field);
      B = B + A * sh;
      const double a[3] = {A.x, A.y, A.z}, gg[3] = {g.x, g.y, g.z};
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) J[i][j] += a[i] * gg[j];
    }
  }
}

// dL/d(field parameters) += (dB(X)/d parameters)^T Bbar: amplitude fields into amp[3 q + i] (a
// per-thread array), grid samples into the field's gradient array with atomics.
__device__ void field_param_vjp(const srs_field *F, int nf, V3 X, V3 Bbar, double *amp, double *const *grid_grads) {
  for (int q = 0; q < nf; ++q) {
    const srs_field &f = F[q];
    if (f.kind == SRS_FIELD_GRID) {
      double *gg = grid_grads ? grid_grads[q] : nullptr;
      if (!gg) continue;
      const AxisCorners one = axis_corners(f, X);
      if (one.axis >= 0) {
        if (one.inside)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            atomicAdd(gg + 3 * (one.k + c) + 0, one.w[c] * Bbar.x);
            atomicAdd(gg + 3 * (one.k + c) + 1, one.w[c] * Bbar.y);
            atomicAdd(gg + 3 * (one.k + c) + 2, one.w[c] * Bbar.z);
          }
        continue;
      }
      Corners C;
      grid_corners(f, X, C);
      for (int c = 0; c < C.nc; ++c) {
        atomicAdd(gg + 3 * C.idx[c] + 0, C.w[c] * Bbar.x);
        atomicAdd(gg + 3 * C.idx[c] + 1, C.w[c] * Bbar.y);
        atomicAdd(gg + 3 * C.idx[c] + 2, C.w[c] * Bbar.z);
      }
    } else if (q < kAdjMaxFields) {
      V3 g;
      const double sh = amp_shape(f, X, g);
      amp[3 * q + 0] += sh * Bbar.x;
      amp[3 * q + 1] += sh * Bbar.y;
      amp[3 * q + 2] += sh * Bbar.z;
    }
  }
}

__device__ inline V3 matvec(const double J[3][3], V3 d) {
  return v3(J[0][0] * d.x + J[0][1] * d.y + J[0][2] * d.z, J[1][0] * d.x + J[1][1] * d.y + J[1][2] * d.z,
            J[2][0] * d.x + J[2][1] * d.y + J[2][2] * d.z);
}
__device__ inline V3 matTvec(const double J[3][3], V3 d) {
  return v3(J[0][0] * d.x + J[1][0] * d.y + J[2][0] * d.z, J[0][1] * d.x + J[1][1] * d.y + J[2][1] * d.z,
            J[0][2] * d.x + J[1][2] * d.y + J[2][2] * d.z);
}

// The four stage states of RK4 step (pos, vel, h), with B and dB/dX at each (same stage structure as
// the forward integrator: OSCARSSR.cc:826-874).
struct Stages {
  V3 p[4], v[4], B[4];
  double J[4][3][3];
};

__device__ void make_stages(const srs_field *F, int nf, double q, V3 pos, V3 vel, double h, Stages &S) {
  const double hh = 0.5 * h;
  S.p[0] = pos;
  S.v[0] = vel;
  field_jet(F, nf, S.p[0], S.B[0], S.J[0]);
  V3 a = cross(S.v[0], S.B[0]) * q;
  S.p[1] = pos + S.v[0] * hh;
  S.v[1] = vel + a * hh;
  field_jet(F, nf, S.p[1], S.B[1], S.J[1]);
  a = cross(S.v[1], S.B[1]) * q;
  S.p[2] = pos + S.v[1] * hh;
  S.v[2] = vel + a * hh;
  field_jet(F, nf, S.p[2], S.B[2], S.J[2]);
  a = cross(S.v[2], S.B[2]) * q;
  S.p[3] = pos + S.v[2] * h;
  S.v[3] = vel + a * h;
  field_jet(F, nf, S.p[3], S.B[3], S.J[3]);
}

// Forward-mode: the tangent (dp, dv, dq) of the step's input -> tangent of its output.
__device__ void step_jvp(const Stages &S, double q, double h, V3 dp, V3 dv, double dq, V3 &odp, V3 &odv) {
  const double hh = 0.5 * h, coef[4] = {0.0, hh, hh, h}, wgt[4] = {1.0, 2.0, 2.0, 1.0};
  V3 sp = dp, sv = dv, accp = v3(0, 0, 0), accv = v3(0, 0, 0), da = v3(0, 0, 0);
  for (int s = 0; s < 4; ++s) {
    if (s > 0) {
      sp = dp + sv * coef[s];  // p_s = pos + coef_s v_{s-1}
      sv = dv + da * coef[s];  // v_s = vel + coef_s a_{s-1}
    }
    da = (cross(S.v[s], S.B[s]) * dq + cross(sv, S.B[s]) * q + cross(S.v[s], matvec(S.J[s], sp)) * q);
    accp = accp + sv * wgt[s];
    accv = accv + da * wgt[s];
  }
  odp = dp + accp * (h / 6.0);
  odv = dv + accv * (h / 6.0);
}

// Reverse-mode: adjoint (lp, lv) of the step's output -> adjoint of its input (pb, vb), q/(m gamma)
// adjoint qb, and the field-parameter contributions.
__device__ void step_vjp(const srs_field *F, int nf, const Stages &S, double q, double h, V3 lp, V3 lv, V3 &pb,
                         V3 &vb, double &qb, double *amp, double *const *grid_grads) {
  const double hh = 0.5 * h, coef[4] = {0.0, hh, hh, h}, wgt[4] = {1.0, 2.0, 2.0, 1.0};
  V3 vbar[4], abar[4];
  for (int s = 0; s < 4; ++s) {
    vbar[s] = lp * (h / 6.0 * wgt[s]);
    abar[s] = lv * (h / 6.0 * wgt[s]);
  }
  pb = lp;
  vb = lv;
  for (int s = 3; s >= 0; --s) {
    // a_s = q v_s x B_s
    vbar[s] = vbar[s] + cross(S.B[s], abar[s]) * q;
    const V3 Bbar = cross(abar[s], S.v[s]) * q;
    qb += dot(abar[s], cross(S.v[s], S.B[s]));
    const V3 pbar = matTvec(S.J[s], Bbar);
    field_param_vjp(F, nf, S.p[s], Bbar, amp, grid_grads);
    pb = pb + pbar;
    vb = vb + vbar[s];
    if (s > 0) {
      abar[s - 1] = abar[s - 1] + vbar[s] * coef[s];
      vbar[s - 1] = vbar[s - 1] + pbar * coef[s];
    }
  }
}

// ---------------------------------------------------------------- chains and scan

struct Chain {
  int64_t L;         // states in the chain (steps: L - 1)
  double h;          // step
  int64_t base;      // stored index of state 0
  int dir;           // stored index of state j: base + dir * j
  int64_t nblk;      // blocks
  int64_t blk_off;   // first global block index
  int64_t step_off;  // first global step index (Jacobian storage)
  int skip_g0;       // state 0's g belongs to the other chain
};
struct Chains {
  Chain c[2];
  int n;
  int64_t total_blocks;
};

struct Traj {
  const double *x, *beta, *gx, *gb;
  int64_t n;
};

__device__ inline void load_state(const Traj &T, int64_t k, V3 &pos, V3 &vel) {
  pos = v3(T.x[k], T.x[T.n + k], T.x[2 * T.n + k]);
  vel = v3(T.beta[k] * kC, T.beta[T.n + k] * kC, T.beta[2 * T.n + k] * kC);
}
// g of chain state j in (x, beta) units
__device__ inline void load_g(const Traj &T, const Chain &ch, int64_t j, double g[6]) {
  if (j == 0 && ch.skip_g0) {
    for (int r = 0; r < 6; ++r) g[r] = 0.0;
    return;
  }
  const int64_t k = ch.base + ch.dir * j;
  for (int c = 0; c < 3; ++c) {
    g[c] = T.gx[c * T.n + k];
    g[3 + c] = T.gb[c * T.n + k];
  }
}

__device__ inline int find_chain(const Chains &C, int64_t block) { return C.n > 1 && block >= C.c[1].blk_off ? 1 : 0; }

// A block's Jacobians in shared memory: step t's 36 entries from jac_at(t).  The odd stride and the extra
// double per chunk keep both the threads' own steps and the chunks' same steps on different banks.
__device__ __forceinline__ int jac_at(int t) { return 37 * t + t / kAdjChunk; }
constexpr int kJacDoubles = 37 * kAdjBlock + kAdjChunks;

// (a) J~_j (6 x 6, row = output, column = input, in (x, beta) units) of every step, and the maps of the
// block's chunks, composed backwards from M = I, b = 0: eight lanes per chunk, one per
// column of M and one for b.  Bound by the latency of the four stages and six tangents of a step with one
// warp per scheduler: 20001 points (157 blocks) 28 us, where the Jacobians (36 us) and then the maps of
// the chunks by one thread each (41 us) took two kernels.
__global__ void __launch_bounds__(kAdjBlock) step_maps_kernel(const srs_field *__restrict__ gF, int nf, double q, Traj T,
                                                              Chains C, double *__restrict__ jac,
                                                              double *__restrict__ chunk_maps) {
  __shared__ double sJ[kJacDoubles];
  __shared__ union {
    srs_field F[kAdjMaxFields];
    struct {
      double g[kAdjBlock][6], map[kAdjChunks][42];
    };
  } sh;
  const int t = threadIdx.x;
  for (int i = t; i < nf; i += kAdjBlock) sh.F[i] = gF[i];
  __syncthreads();
  const Chain &ch = C.c[find_chain(C, blockIdx.x)];
  const int64_t j0 = (blockIdx.x - ch.blk_off) * kAdjBlock;
  const int cnt = (int)imin64(kAdjBlock, ch.L - 1 - j0);
  if (t < cnt) {
    V3 pos, vel;
    load_state(T, ch.base + ch.dir * (j0 + t), pos, vel);
    Stages S;
    make_stages(sh.F, nf, q, pos, vel, ch.h, S);
    double *const Jo = sJ + jac_at(t);
    for (int col = 0; col < 6; ++col) {
      V3 dp = v3(0, 0, 0), dv = v3(0, 0, 0);
      if (col < 3) dp = v3(col == 0, col == 1, col == 2);
      else dv = v3(col == 3, col == 4, col == 5) * kC;
      V3 op, ov;
      step_jvp(S, q, ch.h, dp, dv, 0.0, op, ov);
      const double out[6] = {op.x, op.y, op.z, ov.x / kC, ov.y / kC, ov.z / kC};
      for (int r = 0; r < 6; ++r) Jo[6 * r + col] = out[r];
    }
  }
  __syncthreads();
  if (t < cnt) {
    double g[6];
    load_g(T, ch, j0 + t, g);
    for (int r = 0; r < 6; ++r) sh.g[t][r] = g[r];
  }
  for (int k = t; k < 36 * cnt; k += kAdjBlock) jac[36 * (ch.step_off + j0) + k] = sJ[jac_at(k / 36) + k % 36];
  __syncthreads();
  const int col = t % 8;
  if (t < 8 * kAdjChunks && col < 7) {
    const int c = t / 8;
    double m[6];
    for (int r = 0; r < 6; ++r) m[r] = r == col;
    for (int j = min((c + 1) * kAdjChunk, cnt) - 1; j >= c * kAdjChunk; --j) {
      const double *const J = sJ + jac_at(j);  // lambda_j = g_j + J^T lambda_{j+1}
      double n[6];
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double s = col == 6 ? sh.g[j][r] : 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) s += J[6 * k + r] * m[k];
        n[r] = s;
      }
#pragma unroll
      for (int r = 0; r < 6; ++r) m[r] = n[r];
    }
    for (int r = 0; r < 6; ++r) sh.map[c][col < 6 ? 6 * r + col : 36 + r] = m[r];
  }
  __syncthreads();
  for (int k = t; k < 42 * kAdjChunks; k += kAdjBlock) chunk_maps[42 * kAdjChunks * (int64_t)blockIdx.x + k] = sh.map[k / 42][k % 42];
}

// b + M lambda for row r of an affine map, as a tree (depth 4 instead of a chain of six multiply-adds);
// the six lanes from `first` hold lambda
__device__ __forceinline__ double apply_row(const double m[6], double b, double lam, int first) {
  double l[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) l[k] = __shfl_sync(0xffffffffu, lam, first + k);
  return b + (((m[0] * l[0] + m[1] * l[1]) + (m[2] * l[2] + m[3] * l[3])) + (m[4] * l[4] + m[5] * l[5]));
}

// (b) one warp per chain, lanes 0..5 own one component: lambda at every chunk's end.  Sequential over the chunks;
// the maps come through shared memory in tiles of kCarryTile, the next tile's asynchronous copies in flight
// while the current one is applied, and a map's row is in registers before the map's turn: 95
// us for the 1250 maps of 20001 points (155 when a row was loaded at its turn).  Carrying across maps of whole
// blocks takes 37, but the longitudinal derivative, in which the terms cancel to ~1e-10, then moves by up
// to 1e-9 of the gradient against the carry over these maps (by 3e-10 as it is).
constexpr int kCarryTile = 64;  // chunk maps per tile: 64 x 42 doubles = 21.5 KB, two buffers
__global__ void __launch_bounds__(32) carry_kernel(Traj T, Chains C, const double *__restrict__ chunk_maps,
                                                   double *__restrict__ lam_end) {
  __shared__ __align__(16) double tile[2][kCarryTile * 42];
  const Chain &ch = C.c[blockIdx.x];
  const int r = threadIdx.x, rr = r < 6 ? r : 0;
  if (ch.nblk == 0) return;
  const int64_t nch = (ch.L - 1 + kAdjChunk - 1) / kAdjChunk, off = ch.blk_off * kAdjChunks;
  double g[6];
  load_g(T, ch, ch.L - 1, g);
  double lam = 0.0;  // lambda_{L-1} = g_{L-1}
#pragma unroll
  for (int k = 0; k < 6; ++k)
    if (r == k) lam = g[k];
  const int64_t ntiles = (nch + kCarryTile - 1) / kCarryTile;
  // tile t: the chunks from hi(t) = nch - 1 - t * kCarryTile down to lo(t)
  auto lo_of = [&](int64_t t) { return nch - (t + 1) * kCarryTile > 0 ? nch - (t + 1) * kCarryTile : (int64_t)0; };
  auto fetch = [&](int64_t t) {  // 16-byte copies: a chunk map is 21 of them, 16-byte aligned
    if (t < ntiles) {
      const int64_t lo = lo_of(t);
      const double *const src = chunk_maps + 42 * (off + lo);
      const int n16 = (int)(nch - t * kCarryTile - lo) * 21;
      for (int k = r; k < n16; k += 32) __pipeline_memcpy_async(&tile[t & 1][2 * k], src + 2 * k, 16);
    }
    __pipeline_commit();
  };
  fetch(0);
  for (int64_t t = 0; t < ntiles; ++t) {
    fetch(t + 1);
    __pipeline_wait_prior(1);
    __syncwarp();
    const int64_t lo = lo_of(t);
    int c = (int)(nch - t * kCarryTile - lo) - 1;
    constexpr int kAhead = 4;
    double m[kAhead][7];
    auto load = [&](int k, double *o) {
      const double *const p = tile[t & 1] + 42 * (k > 0 ? k : 0);
#pragma unroll
      for (int q = 0; q < 6; q += 2) {
        const double2 v = *reinterpret_cast<const double2 *>(p + 6 * rr + q);
        o[q] = v.x;
        o[q + 1] = v.y;
      }
      o[6] = p[36 + rr];
    };
#pragma unroll
    for (int a = 0; a < kAhead; ++a) load(c - a, m[a]);
    double *out = lam_end + 6 * (off + lo) + rr;
    for (; c >= 0; c -= kAhead) {
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        if (c - a < 0) break;
        if (r < 6) out[6 * (c - a)] = lam;
        lam = apply_row(m[a], m[a][6], lam, 0);
        load(c - a - kAhead, m[a]);
      }
    }
    __syncwarp();  // every lane is done with this buffer before the next iteration refills it
  }
}

// (c) per block: lambda at the steps' ends, then the reverse-mode step of every step; the field-parameter and q contributions go to per-block partials (amplitudes, q; a fixed tree) or
// atomics (grid samples).  Only the 6 x 6 products of 16 steps are serial; 20001 points 33 us (258 when a
// thread ran the reverse-mode steps of its chunk one after another).
__global__ void __launch_bounds__(kAdjBlock) finish_kernel(const srs_field *__restrict__ gF, int nf, double q, Traj T,
                                                           Chains C, const double *__restrict__ jac,
                                                           const double *__restrict__ lam_end,
                                                           double *const *grid_grads, double *__restrict__ amp_part,
                                                           double *__restrict__ q_part, double *__restrict__ lam_init) {
  __shared__ srs_field F[kAdjMaxFields];
  __shared__ double sJ[kJacDoubles];
  __shared__ double lam_g[kAdjBlock][6];  // g_j, then lambda_{j+1}
  const int t = threadIdx.x, lane = t & 31;
  const int chain = find_chain(C, blockIdx.x);
  const Chain &ch = C.c[chain];
  const int64_t b = blockIdx.x - ch.blk_off, j0 = b * kAdjBlock;
  const int cnt = (int)imin64(kAdjBlock, ch.L - 1 - j0);
  for (int i = t; i < nf; i += kAdjBlock) F[i] = gF[i];
  for (int k = t; k < 36 * cnt; k += kAdjBlock) sJ[jac_at(k / 36) + k % 36] = jac[36 * (ch.step_off + j0) + k];
  V3 pos = v3(0, 0, 0), vel = v3(0, 0, 0);
  if (t < cnt) {
    double g[6];
    load_g(T, ch, j0 + t, g);
    for (int r = 0; r < 6; ++r) lam_g[t][r] = g[r];
    load_state(T, ch.base + ch.dir * (j0 + t), pos, vel);
  }
  __syncthreads();
  if (t < 8 * kAdjChunks) {  // (two whole warps: eight lanes per chunk, six of them one component each)
    const int c = t / 8, r = t % 8 < 6 ? t % 8 : 0;
    double lam = c * kAdjChunk < cnt ? lam_end[6 * (kAdjChunks * (int64_t)blockIdx.x + c) + r] : 0.0;
    for (int j = (c + 1) * kAdjChunk - 1; j >= c * kAdjChunk; --j) {
      const double *const J = sJ + jac_at(j);  // (past the end: not used)
      double m[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) m[k] = J[6 * k + r];
      const double g = lam_g[j][r];
      __syncwarp();
      if (j < cnt && t % 8 < 6) lam_g[j][r] = lam;
      const double next = apply_row(m, g, lam, lane & 24);
      if (j < cnt) lam = next;
    }
    if (t < 6 && b == 0) lam_init[6 * chain + t] = lam;
  }
  __syncthreads();
  double amp[3 * kAdjMaxFields];
  for (int i = 0; i < 3 * nf; ++i) amp[i] = 0.0;
  double qb = 0.0;
  if (t < cnt) {
    const double *const lam = lam_g[t];
    Stages S;
    make_stages(F, nf, q, pos, vel, ch.h, S);
    V3 pb, vb;
    step_vjp(F, nf, S, q, ch.h, v3(lam[0], lam[1], lam[2]), v3(lam[3], lam[4], lam[5]) * (1.0 / kC), pb, vb, qb, amp,
             grid_grads);
  }
  double *const red = sJ;  // (its last readers passed the barrier)
  for (int i = -1; i < 3 * nf; ++i) {
    double v = i < 0 ? qb : amp[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[(i + 1) * (kAdjBlock / 32) + t / 32] = v;
  }
  __syncthreads();
  for (int i = t; i < 1 + 3 * nf; i += kAdjBlock) {
    double v = 0.0;
    for (int w = 0; w < kAdjBlock / 32; ++w) v += red[i * (kAdjBlock / 32) + w];
    if (i == 0) q_part[blockIdx.x] = v;
    else amp_part[(int64_t)3 * nf * blockIdx.x + i - 1] = v;
  }
}

// Fixed-order totals: out[0..2] dL/dx0, out[3..5] dL/dbeta0, out[6] dL/dq, out[7..] amplitudes.  The
// per-block partials of q and of each amplitude are added by the block: thread t adds a contiguous
// run of them in order, then a fixed tree over the 128 runs (a deterministic order).
__global__ void __launch_bounds__(128) adjoint_total_kernel(Chains C, int nf, const double *__restrict__ lam_init,
                                                            const double *__restrict__ amp_part,
                                                            const double *__restrict__ q_part,
                                                            double *__restrict__ out) {
  __shared__ double red[128];
  const int t = threadIdx.x;
  if (t < 6) {
    double s = 0.0;
    for (int k = 0; k < C.n; ++k) s += lam_init[6 * k + t];
    out[t] = s;
  }
  const int64_t total = C.total_blocks, per = (total + 127) / 128;
  const int64_t g0 = t * per, g1 = g0 + per < total ? g0 + per : total;
  for (int o = 0; o < 1 + 3 * nf; ++o) {  // o = 0: q; o = 1 + i: amplitude i
    double s = 0.0;
    for (int64_t g = g0; g < g1; ++g) s += o == 0 ? q_part[g] : amp_part[(int64_t)3 * nf * g + (o - 1)];
    red[t] = s;
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
      if (t < w) red[t] += red[t + w];
      __syncthreads();
    }
    if (t == 0) out[6 + o] = red[0];
    __syncthreads();
  }
}

// ---------------------------------------------------------------- sum adjoint

// Per energy k, nine doubles: w_k, 2 w conj(E_k) with w = dL/dflux_k * C2 (C0 w_k dt)^2, c/w_k, w_k/c.
constexpr int kWeightDoubles = 9;  // (odd: four energies side by side in shared memory are on different banks)
__global__ void spectrum_weights_kernel(const double *__restrict__ energies, const double *__restrict__ e6,
                                        const double *__restrict__ gflux, int64_t ne, double dt, double C0, double C2,
                                        double *__restrict__ W) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ne) return;
  const double om = ev_to_omega(energies[k]);
  const double g = C0 * om * dt;
  const double w = 2.0 * gflux[k] * C2 * g * g;
  W += kWeightDoubles * k;
  W[0] = om;
  W[7] = kC / om;
  W[8] = om / kC;
  for (int c = 0; c < 3; ++c) {
    W[1 + 2 * c] = w * e6[6 * k + 2 * c];
    W[2 + 2 * c] = -w * e6[6 * k + 2 * c + 1];
  }
}

// kSumAdjLanes lanes share a point, each every kSumAdjLanes-th energy: a trajectory has too few points for one
// thread each (20001: one warp per scheduler).  Only the three sums that the derivatives are linear in are
// formed per energy: ~50 operations, where the derivatives themselves took ~220 with two divisions;
// 20001 points x 200 energies 90 -> 28 us (12 at the FP64 pipe's rate).
constexpr int kSumAdjThreads = 128, kSumAdjTile = 128, kSumAdjLanes = 4, kSumAdjPoints = kSumAdjThreads / kSumAdjLanes;

__global__ void __launch_bounds__(kSumAdjThreads) spectrum_adjoint_kernel(const double *__restrict__ X,
                                                                          const double *__restrict__ Bt, int64_t n,
                                                                          double dt, V3 obs,
                                                                          const double *__restrict__ W, int64_t ne,
                                                                          double *__restrict__ gx,
                                                                          double *__restrict__ gb) {
  __shared__ double sW[kSumAdjTile * kWeightDoubles];
  const int64_t i = (int64_t)blockIdx.x * kSumAdjPoints + threadIdx.x / kSumAdjLanes;
  const bool active = i < n;
  const int64_t ii = active ? i : n - 1;
  const V3 x = v3(X[ii], X[n + ii], X[2 * n + ii]);
  const V3 be = v3(Bt[ii], Bt[n + ii], Bt[2 * n + ii]);
  // D, n and the retarded time exactly as the plain FP64 sum forms them (this file is compiled
  // without FMA contraction): the phases w tau are ~1e10 rad, and the adjoint's e^{i w tau} must be
  // the forward's own to the last bit, or the gradient along the trajectory (the near-invariant
  // longitudinal direction, where the per-point terms cancel to ~1e-10) is lost in phase noise.
  const V3 R = obs - x;
  const double D = mag(R), iD = 1.0 / D;
  const V3 nv = R / D;
  const double tau = dt * (double)(int)ii + D / kC;
  const double nn[3] = {nv.x, nv.y, nv.z}, bb[3] = {be.x, be.y, be.z};
  // With P = W e^{i w tau}: A = Sum Re P, Bc = Sum (c/w) Im P, Wc = Sum (w/c) Im P; the derivatives of the
  // amplitude and of the phase are linear in them
  double A[3] = {0, 0, 0}, Bc[3] = {0, 0, 0}, Wc[3] = {0, 0, 0};
  __shared__ BlockBound longest;  // the retarded times
  longest.set(tau);
  for (int64_t k0 = 0; k0 < ne; k0 += kSumAdjTile) {
    const int cnt = (int)imin64(kSumAdjTile, ne - k0);
    __syncthreads();
    bool far = false;
    for (int t = threadIdx.x; t < cnt * kWeightDoubles; t += blockDim.x) {
      const double v = W[kWeightDoubles * k0 + t];
      sW[t] = v;
      if (t % kWeightDoubles == 0) far = far || phases_far(v, longest.get());
    }
    far = __syncthreads_or(far);
    auto term = [&](int k, auto is_far) {
      const double *const w = sW + kWeightDoubles * k;
      double sn, cs;
      sincos_phase<is_far.value>(w[0] * tau, sn, cs);
      const double cow = w[7], woc = w[8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double wr = w[1 + 2 * c], wi = w[2 + 2 * c];
        const double pi = __fma_rn(wr, sn, wi * cs);
        A[c] += __fma_rn(wr, cs, -(wi * sn));
        Bc[c] = __fma_rn(cow, pi, Bc[c]);
        Wc[c] = __fma_rn(woc, pi, Wc[c]);
      }
    };
    if (far)
      for (int k = threadIdx.x % kSumAdjLanes; k < cnt; k += kSumAdjLanes) term(k, std::true_type{});
    else
      for (int k = threadIdx.x % kSumAdjLanes; k < cnt; k += kSumAdjLanes) term(k, std::false_type{});
  }
#pragma unroll
  for (int o = 1; o < kSumAdjLanes; o *= 2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      A[c] += __shfl_xor_sync(0xffffffffu, A[c], o);
      Bc[c] += __shfl_xor_sync(0xffffffffu, Bc[c], o);
      Wc[c] += __shfl_xor_sync(0xffffffffu, Wc[c], o);
    }
  }
  if (!active || threadIdx.x % kSumAdjLanes != 0) return;
  const double iD2 = iD * iD, iD3 = iD2 * iD;
  double Tt = 0.0;
  for (int c = 0; c < 3; ++c)
    Tt += A[c] * (bb[c] - 3.0 * nn[c]) * iD2 + 3.0 * Bc[c] * nn[c] * iD3 + Wc[c] * (bb[c] - nn[c]) * iD;
  for (int c = 0; c < 3; ++c) {
    gb[c * n + i] = A[c] * iD;
    gx[c * n + i] = A[c] * iD2 - Bc[c] * iD3 + nn[c] * Tt;
  }
}

}  // namespace
}  // namespace srs

using namespace srs;

extern "C" {

srs_status srs_spectrum_efield(srs_traj_view traj, srs_beam_consts beam, const double obs[3],
                               const double *d_energies, int64_t ne, int32_t precision, double *d_flux,
                               double *d_e6, void *stream) {
  clear_error();
  if (!traj.x || !traj.beta || traj.n < 1 || traj.nparticles < 1 || !(traj.dt > 0))
    return fail(SRS_ERR_INVALID, "bad trajectory view");
  if (!obs || !d_energies || !d_flux || !d_e6 || ne < 1) return fail(SRS_ERR_INVALID, "bad argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DeviceBuffer scratch;
  if (precision == SRS_PRECISION_FP64) {
    SRS_CUDA(scratch.alloc(fp64_spectrum_scratch_bytes(traj.n, ne, traj.nparticles), s));
    SRS_CUDA(fp64_spectrum(traj, beam, obs, d_energies, ne, d_flux, scratch.ptr, s, d_e6));
  } else if (precision == SRS_PRECISION_MIXED) {
    SRS_CUDA(scratch.alloc(mixed_spectrum_scratch_bytes(traj.n, ne, traj.nparticles), s));
    SRS_CUDA(mixed_spectrum(traj, beam, obs, d_energies, ne, d_flux, scratch.ptr, s, d_e6));
  } else {
    return fail(SRS_ERR_INVALID, "unknown precision");
  }
  return SRS_OK;
}

srs_status srs_spectrum_adjoint(srs_traj_view traj, srs_beam_consts beam, const double obs[3],
                                const double *d_energies, int64_t ne, const double *d_e6, const double *d_gflux,
                                double *d_gx, double *d_gbeta, void *stream) {
  clear_error();
  if (!traj.x || !traj.beta || traj.n < 1 || !(traj.dt > 0)) return fail(SRS_ERR_INVALID, "bad trajectory view");
  if (traj.nparticles != 1) return fail(SRS_ERR_INVALID, "the spectrum adjoint takes one particle");
  if (!obs || !d_energies || !d_e6 || !d_gflux || !d_gx || !d_gbeta || ne < 1)
    return fail(SRS_ERR_INVALID, "bad argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DeviceBuffer W;
  SRS_CUDA(W.alloc(sizeof(double) * kWeightDoubles * ne, s));
  spectrum_weights_kernel<<<(unsigned)((ne + 127) / 128), 128, 0, s>>>(
      d_energies, d_e6, d_gflux, ne, traj.dt, flux_c0(beam.charge), flux_c2(beam.charge, beam.current), W.as<double>());
  SRS_CUDA(cudaGetLastError());
  spectrum_adjoint_kernel<<<(unsigned)((traj.n + kSumAdjPoints - 1) / kSumAdjPoints), kSumAdjThreads, 0, s>>>(
      traj.x, traj.beta, traj.n, traj.dt, v3(obs[0], obs[1], obs[2]), W.as<double>(), ne, d_gx, d_gbeta);
  SRS_CUDA(cudaGetLastError());
  return SRS_OK;
}

srs_status srs_trajectory_adjoint(const srs_field *fields, int32_t nfields, const srs_particle *particle,
                                  double ctstart, double ctstop, double t0, int64_t npoints, const double *d_x,
                                  const double *d_beta, const double *d_gx, const double *d_gbeta,
                                  double *const *grid_grads, double *amp_grad, double *ic_grad, void *stream) {
  clear_error();
  if (!particle || !d_x || !d_beta || !d_gx || !d_gbeta || !ic_grad) return fail(SRS_ERR_INVALID, "NULL argument");
  if (nfields < 0 || nfields > kAdjMaxFields || (nfields > 0 && !fields))
    return fail(SRS_ERR_INVALID, "the adjoint takes 0.." + std::to_string(kAdjMaxFields) + " fields");
  if (has_electric(fields, nfields)) return fail(SRS_ERR_INVALID, "the adjoint takes magnetic fields only");
  double dt;
  int64_t nf, nb;
  if (srs_status st = srs_trajectory_counts(ctstart, ctstop, t0, npoints, &dt, &nf, &nb)) return st;
  if (nf < 1) return fail(SRS_ERR_INVALID, "empty forward trajectory");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Chains C;
  std::memset(&C, 0, sizeof C);
  int64_t blocks = 0, steps = 0;
  auto add = [&](int64_t L, double h, int64_t base, int dir, int skip) {
    Chain &ch = C.c[C.n++];
    ch.L = L;
    ch.h = h;
    ch.base = base;
    ch.dir = dir;
    ch.skip_g0 = skip;
    ch.nblk = (L - 1 + kAdjBlock - 1) / kAdjBlock;
    ch.blk_off = blocks;
    ch.step_off = steps;
    blocks += ch.nblk;
    steps += L - 1;
  };
  add(nf, dt, nb, +1, 0);
  if (nb > 0) add(nb + 1, -dt, nb, -1, 1);
  C.total_blocks = blocks;
  const Traj T{d_x, d_beta, d_gx, d_gbeta, nf + nb};
  const double q = particle->qomg;

  // device copies: fields, grid-gradient pointer table
  DeviceBuffer dF, dG, jac, Mb, lam, amp, qp, laminit, out;
  SRS_CUDA(dF.alloc(sizeof(srs_field) * std::max(1, nfields), s));
  SRS_CUDA(dG.alloc(sizeof(double *) * std::max(1, nfields), s));
  std::vector<double *> gg(std::max(1, nfields), nullptr);
  for (int i = 0; i < nfields; ++i) gg[i] = grid_grads ? grid_grads[i] : nullptr;
  if (nfields > 0)
    SRS_CUDA(cudaMemcpyAsync(dF.ptr, fields, sizeof(srs_field) * nfields, cudaMemcpyHostToDevice, s));
  SRS_CUDA(cudaMemcpyAsync(dG.ptr, gg.data(), sizeof(double *) * gg.size(), cudaMemcpyHostToDevice, s));
  const int64_t nb1 = std::max<int64_t>(1, blocks);
  SRS_CUDA(jac.alloc(sizeof(double) * 36 * std::max<int64_t>(1, steps), s));
  SRS_CUDA(Mb.alloc(sizeof(double) * 42 * kAdjChunks * nb1, s));
  SRS_CUDA(lam.alloc(sizeof(double) * 6 * kAdjChunks * nb1, s));
  SRS_CUDA(amp.alloc(sizeof(double) * 3 * std::max(1, nfields) * nb1, s));
  SRS_CUDA(qp.alloc(sizeof(double) * nb1, s));
  SRS_CUDA(laminit.alloc(sizeof(double) * 12, s));
  SRS_CUDA(out.alloc(sizeof(double) * (7 + 3 * std::max(1, nfields)), s));
  SRS_CUDA(cudaMemsetAsync(laminit.ptr, 0, sizeof(double) * 12, s));
  const srs_field *Fd = dF.as<srs_field>();
  if (steps > 0) {
    step_maps_kernel<<<(unsigned)blocks, kAdjBlock, 0, s>>>(Fd, nfields, q, T, C, jac.as<double>(), Mb.as<double>());
    SRS_CUDA(cudaGetLastError());
    carry_kernel<<<C.n, 32, 0, s>>>(T, C, Mb.as<double>(), lam.as<double>());
    SRS_CUDA(cudaGetLastError());
    finish_kernel<<<(unsigned)blocks, kAdjBlock, 0, s>>>(Fd, nfields, q, T, C, jac.as<double>(),
                                                         lam.as<double>(), reinterpret_cast<double *const *>(dG.ptr),
                                                         amp.as<double>(), qp.as<double>(), laminit.as<double>());
    SRS_CUDA(cudaGetLastError());
  }
  // chains of a single state: lambda_0 = g_0
  for (int k = 0; k < C.n; ++k)
    if (C.c[k].L == 1 && !C.c[k].skip_g0) {
      for (int c = 0; c < 3; ++c) {
        SRS_CUDA(cudaMemcpyAsync(laminit.as<double>() + 6 * k + c, d_gx + c * T.n + C.c[k].base, sizeof(double),
                                 cudaMemcpyDeviceToDevice, s));
        SRS_CUDA(cudaMemcpyAsync(laminit.as<double>() + 6 * k + 3 + c, d_gbeta + c * T.n + C.c[k].base,
                                 sizeof(double), cudaMemcpyDeviceToDevice, s));
      }
    }
  adjoint_total_kernel<<<1, 128, 0, s>>>(C, nfields, laminit.as<double>(), amp.as<double>(), qp.as<double>(),
                                         out.as<double>());
  SRS_CUDA(cudaGetLastError());
  std::vector<double> h(7 + 3 * std::max(1, nfields));
  SRS_CUDA(cudaMemcpyAsync(h.data(), out.ptr, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
  SRS_CUDA(cudaStreamSynchronize(s));
  for (int i = 0; i < 7; ++i) ic_grad[i] = h[i];
  if (amp_grad)
    for (int i = 0; i < 3 * nfields; ++i) amp_grad[i] = h[7 + i];
  return SRS_OK;
}

}  // extern "C"
