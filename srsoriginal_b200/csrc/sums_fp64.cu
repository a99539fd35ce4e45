// Plain FP64 radiation sums: the drop-in for the reference's GPU/CPU sums (this file is compiled with
// -fmad=false; fused operations are written out).
//
//   spectrum  : OSCARSSR::CalculateSpectrum   src/OSCARSSR.cc:1154-1251 (energy loop :1202-1246)
//   flux      : OSCARSSR::CalculateFlux2      src/OSCARSSR.cc:1989-2099 (point loop :2054-2096)
//   power dens: OSCARSSR::CalculatePowerDensity src/OSCARSSR.cc:1477-1598 (loop :1533-1560)
//   total pow : OSCARSSR::CalculateTotalPower src/OSCARSSR.cc:1939-1978
//
// Per term the flux/spectrum integrand is (beta - n (1 + i c/(w D)))/D exp(i w (i dt + D/c)), summed
// over trajectory points.  What decides the result's bits is kept in the reference's IEEE operation
// order: D = RN(sqrt(|R|^2)) and the phase w*(i*dt + D/c) (~1e11 rad: one rounding of it moves a
// term by ~1e-5 rad), and for the power density n = R/D and 1 - n.beta (~1e-8, raised to the fifth
// power).  Everything after them only carries relative errors of ~1e-16 into the term, so it is
// arranged for the FP64 pipe, which bounds these kernels (a fused multiply-add is one operation):
//  * D, 1/D and the quotients by D from one reciprocal square root (sqrt_both, div_rn): no division
//    sequence;
//  * the phase reduced to |r| <= pi/4 in four operations and its sine and cosine from two polynomials
//    (sincos_reduced): 20 operations per term;
//  * the near-field term i c/(w D) n/D and the factor 1/D applied to the phasor instead of to the six
//    amplitude components, the sums as fused multiply-adds;
//  * the power density's |V|^2 as the sum of V's squared components (V is perpendicular to n, so the
//    reference's two projections on a basis normal to n add up to it).
// Operations per term: flux 63, spectrum 33, power density 63 (127, ~75 and ~165 when every step was in
// the reference's order).
//
// Parallel layout (B200: 148 SMs): one thread per output (energy or observation point), 128 outputs
// per CTA, and the trajectory axis split into S contiguous chunks across CTAs so that small outputs
// (1000 energies) still fill every SM.  Each CTA stages its chunk through shared memory in 128-point
// tiles, read by all threads as broadcasts.  Partial complex sums go to scratch, and a second kernel
// adds the S partials in chunk order (deterministic) and applies the reference's final scaling.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "splits.h"
#include "srs_device.cuh"
#include "srs_internal.h"

namespace srs {

namespace {

constexpr int kTile = 128;     // outputs per CTA and trajectory points per shared-memory tile

// Trajectory points per CTA for `ctas` tiles of outputs: the split of least waves * (points + overhead)
// over the launches of up to six full waves, in multiples of 32 points (a small output then still
// spreads over the GPU).
int64_t chunk_for(int64_t ctas, int64_t n, int64_t slots) {
  constexpr int64_t kGranule = 32, kOverhead = 24;
  int64_t best = n, best_cost = INT64_MAX;
  for (int64_t w = 1; w <= 6; ++w) {
    const int64_t s = std::min<int64_t>(std::max<int64_t>(1, w * slots / std::max<int64_t>(1, ctas)), 65535);
    int64_t chunk = ((n + s - 1) / s + kGranule - 1) / kGranule * kGranule;
    chunk = std::max(chunk, (n + 65534) / 65535);
    const int64_t used = (n + chunk - 1) / chunk, waves = (ctas * used + slots - 1) / slots;
    const int64_t cost = waves * (chunk + kOverhead);
    if (cost < best_cost) {
      best_cost = cost;
      best = chunk;
    }
  }
  return best;
}

// ---------------------------------------------------------------- flux at observation points

__global__ void __launch_bounds__(kTile) flux_fp64_kernel(const double *__restrict__ X, const double *__restrict__ Bt,
                                                          int64_t n, double dt, const double *__restrict__ pts,
                                                          int64_t np, double omega, int64_t chunk,
                                                          double *__restrict__ partial) {
  static_assert(kTile == 128, "BlockBound's four warps");
  __shared__ double2 tile[4][kTile];  // (x, y), (z, i dt), (beta_x, beta_y), (beta_z, -)
  wait_for_previous_grid();  // (launched with launch_after)
  allow_next_grid();
  const int tid = threadIdx.x;
  const int64_t j = (int64_t)blockIdx.x * kTile + tid;
  const int s = blockIdx.y, S = gridDim.y, p = blockIdx.z;
  const double *xp = X + (int64_t)p * 3 * n, *bp = Bt + (int64_t)p * 3 * n;
  const int64_t i0 = (int64_t)s * chunk, i1 = imin64(n, i0 + chunk);
  const bool active = j < np;
  V3 obs = active ? v3(pts[3 * j], pts[3 * j + 1], pts[3 * j + 2]) : v3(0, 0, 1);
  const double icow = kC / omega, rc = 1.0 / kC;
  __shared__ BlockBound reach;  // of the block's points (no distance exceeds |x| + |y| + |z| of both ends)
  reach.set(fabs(obs.x) + fabs(obs.y) + fabs(obs.z));
  double axr = 0, axi = 0, ayr = 0, ayi = 0, azr = 0, azi = 0;
  for (int64_t base = i0; base < i1; base += kTile) {
    const int cnt = (int)imin64(kTile, i1 - base);
    __syncthreads();
    bool far = false;
    if (tid < cnt) {
      const int64_t i = base + tid;
      const V3 x = v3(xp[i], xp[n + i], xp[2 * n + i]);
      const double t = dt * (double)(int)i;
      tile[0][tid] = make_double2(x.x, x.y);
      tile[1][tid] = make_double2(x.z, t);
      tile[2][tid] = make_double2(bp[i], bp[n + i]);
      tile[3][tid] = make_double2(bp[2 * n + i], 0.0);
      far = phases_far(omega, fabs(t) + (fabs(x.x) + fabs(x.y) + fabs(x.z) + reach.get()) * rc);
    }
    far = __syncthreads_or(far);
    if (!active) continue;
    auto term = [&](int k, auto is_far) {
      const double2 q0 = tile[0][k], q1 = tile[1][k], q2 = tile[2][k];
      const double bz = tile[3][k].x;
      const V3 R = obs - v3(q0.x, q0.y, q1.x);
      double m, y, sn, cs;
      sqrt_both(mag2(R), m, y);
      sincos_phase<is_far.value>(omega * (q1.y + div_rn(m, kC, rc)), sn, cs);
      // (beta - n)/D e^{i phi} - i (c/w) n/D^2 e^{i phi}, with e^{i phi}/D = (cr, ci)
      const double cr = y * cs, ci = y * sn, f = icow * y * y, fr = f * cr, fi = f * ci;
      const double dx = __fma_rn(-R.x, y, q2.x), dy = __fma_rn(-R.y, y, q2.y), dz = __fma_rn(-R.z, y, bz);
      axr = __fma_rn(dx, cr, __fma_rn(R.x, fi, axr));
      axi = __fma_rn(dx, ci, __fma_rn(-R.x, fr, axi));
      ayr = __fma_rn(dy, cr, __fma_rn(R.y, fi, ayr));
      ayi = __fma_rn(dy, ci, __fma_rn(-R.y, fr, ayi));
      azr = __fma_rn(dz, cr, __fma_rn(R.z, fi, azr));
      azi = __fma_rn(dz, ci, __fma_rn(-R.z, fr, azi));
    };
    if (far) {
#pragma unroll 1
      for (int k = 0; k < cnt; ++k) term(k, std::true_type{});
    } else {
#pragma unroll 2
      for (int k = 0; k < cnt; ++k) term(k, std::false_type{});
    }
  }
  if (active) {
    double *o = partial + ((int64_t)p * S + s) * 6 * np + j;
    o[0] = axr; o[np] = axi; o[2 * np] = ayr; o[3 * np] = ayi; o[4 * np] = azr; o[5 * np] = azi;
  }
}


// Adds the S per-chunk partials of every output and applies the final scaling.  A block holds P outputs x 6
// components x G groups of consecutive chunks: thread (g, c, k) adds its group's chunks of component c of
// output k in chunk order, eight loads in flight, then the groups are added in order (a fixed order).  The
// time is the latency of a thread's batches of loads, so few outputs take more groups: 101 energies in
// 626 chunks 28 -> 5 us, 1000 in 157 9 -> 5 us, against one thread per component.
template <int P, int G>
__global__ void __launch_bounds__(6 * P * G) flux_reduce_kernel(const double *__restrict__ partial, int S, int64_t np,
                                                                int nparticles, const double *__restrict__ omegas,
                                                                const double *__restrict__ energies, double omega0,
                                                                double dt, double C0, double C2,
                                                                double *__restrict__ out, double *__restrict__ e6) {
  __shared__ double se[G][6][P];
  wait_for_previous_grid();  // (launched with launch_after by finish_flux_partials)
  const int k = threadIdx.x % P, c = threadIdx.x / P % 6, g = threadIdx.x / (6 * P);
  const int64_t idx = (int64_t)blockIdx.x * P + k;
  const bool valid = idx < np * nparticles;
  double e = 0;
  if (valid) {
    const int64_t p = idx / np, j = idx % np, stride = 6 * np;
    const int per = (S + G - 1) / G, s0 = g * per, s1 = min(S, s0 + per);
    const double *o = partial + ((p * S + s0) * 6 + c) * np + j;
    int s = s0;
    for (; s + 8 <= s1; s += 8, o += 8 * stride) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = o[u * stride];
#pragma unroll
      for (int u = 0; u < 8; ++u) e += v[u];
    }
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = s + u < s1 ? o[u * stride] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) e += v[u];
  }
  se[g][c][k] = e;
  __syncthreads();
  if (threadIdx.x < P && valid) {
    double t[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      t[q] = se[0][q][k];
#pragma unroll
      for (int u = 1; u < G; ++u) t[q] += se[u][q][k];
    }
    const double omega = energies ? ev_to_omega(energies[idx % np]) : omegas ? omegas[idx % np] : omega0;
    out[idx] = finish_flux(t, omega, dt, C0, C2);
    if (e6) {
#pragma unroll
      for (int q = 0; q < 6; ++q) e6[6 * idx + q] = t[q];
    }
  }
}

// ---------------------------------------------------------------- spectrum at one observer

__global__ void __launch_bounds__(kTile) spectrum_fp64_kernel(const double *__restrict__ X,
                                                              const double *__restrict__ Bt, int64_t n, double dt,
                                                              V3 obs, const double *__restrict__ energies,
                                                              int64_t ne, int64_t chunk,
                                                              double *__restrict__ partial) {
  // Per trajectory point (energy independent): tau = i*dt + D/c, a = (beta - n)/D, b = n/D^2, as
  // (tau, a_x), (a_y, a_z), (b_x, b_y), (b_z, -).  The near-field part -i (c/w) sum b e^{i w tau} is summed
  // without its factor, which is applied once per chunk.
  __shared__ double2 tile[4][kTile];
  wait_for_previous_grid();  // (launched with launch_after)
  allow_next_grid();
  const int tid = threadIdx.x;
  const int64_t k = (int64_t)blockIdx.x * kTile + tid;
  const int s = blockIdx.y, S = gridDim.y, p = blockIdx.z;
  const double *xp = X + (int64_t)p * 3 * n, *bp = Bt + (int64_t)p * 3 * n;
  const int64_t i0 = (int64_t)s * chunk, i1 = imin64(n, i0 + chunk);
  const bool active = k < ne;
  const double omega = active ? ev_to_omega(energies[k]) : 1.0;
  const double icow = kC / omega;
  __shared__ BlockBound top;  // the angular frequencies
  top.set(omega);
  double a[6] = {0, 0, 0, 0, 0, 0}, b[6] = {0, 0, 0, 0, 0, 0};
  for (int64_t base = i0; base < i1; base += kTile) {
    const int cnt = (int)imin64(kTile, i1 - base);
    __syncthreads();
    bool far = false;
    if (tid < cnt) {
      const int64_t i = base + tid;
      const V3 R = obs - v3(xp[i], xp[n + i], xp[2 * n + i]);
      double m, y;
      sqrt_both(mag2(R), m, y);
      const double y2 = y * y, y3 = y2 * y, tau = dt * (double)(int)i + div_rn(m, kC, 1.0 / kC);
      far = phases_far(top.get(), tau);
      tile[0][tid] = make_double2(tau, __fma_rn(-R.x, y, bp[i]) * y);
      tile[1][tid] = make_double2(__fma_rn(-R.y, y, bp[n + i]) * y, __fma_rn(-R.z, y, bp[2 * n + i]) * y);
      tile[2][tid] = make_double2(R.x * y3, R.y * y3);
      tile[3][tid] = make_double2(R.z * y3, 0.0);
    }
    far = __syncthreads_or(far);
    if (!active) continue;
    auto term = [&](int q, auto is_far) {
      const double2 q0 = tile[0][q], q1 = tile[1][q], q2 = tile[2][q];
      const double bz = tile[3][q].x;
      double sn, cs;
      sincos_phase<is_far.value>(omega * q0.x, sn, cs);
      a[0] = __fma_rn(q0.y, cs, a[0]); a[1] = __fma_rn(q0.y, sn, a[1]);
      a[2] = __fma_rn(q1.x, cs, a[2]); a[3] = __fma_rn(q1.x, sn, a[3]);
      a[4] = __fma_rn(q1.y, cs, a[4]); a[5] = __fma_rn(q1.y, sn, a[5]);
      b[0] = __fma_rn(q2.x, cs, b[0]); b[1] = __fma_rn(q2.x, sn, b[1]);
      b[2] = __fma_rn(q2.y, cs, b[2]); b[3] = __fma_rn(q2.y, sn, b[3]);
      b[4] = __fma_rn(bz, cs, b[4]); b[5] = __fma_rn(bz, sn, b[5]);
    };
    if (far) {
#pragma unroll 1
      for (int q = 0; q < cnt; ++q) term(q, std::true_type{});
    } else {
#pragma unroll 2
      for (int q = 0; q < cnt; ++q) term(q, std::false_type{});
    }
  }
  if (active) {
    double *o = partial + ((int64_t)p * S + s) * 6 * ne + k;
#pragma unroll
    for (int c = 0; c < 6; c += 2) {
      o[c * ne] = __fma_rn(icow, b[c + 1], a[c]);
      o[(c + 1) * ne] = __fma_rn(-icow, b[c], a[c + 1]);
    }
  }
}

// ---------------------------------------------------------------- power density

__global__ void __launch_bounds__(kTile) pd_fp64_kernel(const double *__restrict__ X, const double *__restrict__ Bt,
                                                        const double *__restrict__ A, int64_t n,
                                                        const double *__restrict__ pts,
                                                        const double *__restrict__ nrms, int64_t np,
                                                        int directional, int64_t chunk,
                                                        double *__restrict__ partial) {
  __shared__ double2 tile[5][kTile];  // (x, y), (z, beta_x), (beta_y, beta_z), (a_x, a_y), (a_z, -)
  wait_for_previous_grid();  // (launched with launch_after)
  allow_next_grid();
  const int tid = threadIdx.x;
  const int64_t j = (int64_t)blockIdx.x * kTile + tid;
  const int s = blockIdx.y, S = gridDim.y, p = blockIdx.z;
  const int64_t off = (int64_t)p * 3 * n;
  const double *xp = X + off, *bp = Bt + off, *ap = A + off;
  const int64_t i0 = (int64_t)s * chunk, i1 = imin64(n, i0 + chunk);
  const bool active = j < np;
  V3 obs = active ? v3(pts[3 * j], pts[3 * j + 1], pts[3 * j + 2]) : v3(0, 0, 1);
  V3 nrm = active ? v3(nrms[3 * j], nrms[3 * j + 1], nrms[3 * j + 2]) : v3(0, 0, 1);
  double sum = 0;
  // a x b with one rounding less per component
  auto fcross = [](V3 a, V3 b) {
    return v3(__fma_rn(a.y, b.z, -(b.y * a.z)), __fma_rn(a.z, b.x, -(b.z * a.x)), __fma_rn(a.x, b.y, -(b.x * a.y)));
  };
  for (int64_t base = i0; base < i1; base += kTile) {
    const int cnt = (int)imin64(kTile, i1 - base);
    __syncthreads();
    if (tid < cnt) {
      const int64_t i = base + tid;
      tile[0][tid] = make_double2(xp[i], xp[n + i]);
      tile[1][tid] = make_double2(xp[2 * n + i], bp[i]);
      tile[2][tid] = make_double2(bp[n + i], bp[2 * n + i]);
      tile[3][tid] = make_double2(ap[i], ap[n + i]);
      tile[4][tid] = make_double2(ap[2 * n + i], 0.0);
    }
    __syncthreads();
    if (!active) continue;
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
      const double2 q0 = tile[0][k], q1 = tile[1][k], q2 = tile[2][k], q3 = tile[3][k];
      const V3 B = v3(q1.y, q2.x, q2.y), AC = v3(q3.x, q3.y, tile[4][k].x);
      const V3 R = obs - v3(q0.x, q0.y, q1.x);
      const double m2 = mag2(R);
      double m, y;
      sqrt_both(m2, m, y);
      const V3 N = v3(div_rn(R.x, m, y), div_rn(R.y, m, y), div_rn(R.z, m, y));  // RN(R / D)
      const double nd = __fma_rn(N.z, nrm.z, __fma_rn(N.y, nrm.y, N.x * nrm.x));
      const V3 V = fcross(N, fcross(N - B, AC));
      const double omb = 1 - dot(B, N), omb2 = omb * omb;
      const double den = omb2 * omb2 * (omb * m2);
      const double v2 = __fma_rn(V.z, V.z, __fma_rn(V.y, V.y, V.x * V.x));
      const double with = __fma_rn(v2 * nd, reciprocal(den), sum);
      sum = directional && nd <= 0 ? sum : with;
    }
  }
  if (active) partial[((int64_t)p * S + s) * np + j] = sum;
}

// The same for the power density: P outputs x G groups of chunks.
template <int P, int G>
__global__ void __launch_bounds__(P * G) pd_reduce_kernel(const double *__restrict__ partial, int S, int64_t np,
                                                          int nparticles, double cdt, int directional,
                                                          double *__restrict__ out) {
  __shared__ double se[G][P];
  wait_for_previous_grid();  // (launched with launch_after by finish_pd_partials)
  const int k = threadIdx.x % P, g = threadIdx.x / P;
  const int64_t idx = (int64_t)blockIdx.x * P + k;
  const bool valid = idx < np * nparticles;
  double sum = 0;
  if (valid) {
    const int64_t p = idx / np, j = idx % np;
    const int per = (S + G - 1) / G, s0 = g * per, s1 = min(S, s0 + per);
    const double *o = partial + (p * S + s0) * np + j;
    for (int s = s0; s < s1; s += 8, o += 8 * np) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = s + u < s1 ? o[u * np] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) sum += v[u];
    }
  }
  se[g][k] = sum;
  __syncthreads();
  if (g != 0 || !valid) return;
#pragma unroll
  for (int u = 1; u < G; ++u) sum += se[u][k];
  sum *= cdt;
  sum /= 1e6;
  if (!directional && sum < 0) sum *= -1;
  out[idx] = sum;
}

// ---------------------------------------------------------------- total power and accumulation

// One block per particle; the terms (which cancel to 1/gamma^2) in the reference's operation order, their
// sum over points strided over the threads and then over the block in a fixed order (one thread per
// particle took 1.3 ms for 12001 points, this 8 us).
constexpr int kPowerThreads = 512;
__global__ void __launch_bounds__(kPowerThreads) total_power_kernel(const double *__restrict__ Bt,
                                                                    const double *__restrict__ A, int64_t n, double dt,
                                                                    double qi, const double *__restrict__ gamma,
                                                                    double *__restrict__ out) {
  __shared__ double sum[kPowerThreads];
  const int p = blockIdx.x, t = threadIdx.x;
  const double *bp = Bt + (int64_t)p * 3 * n, *ap = A + (int64_t)p * 3 * n;
  double tp = 0;
#pragma unroll 4
  for (int64_t i = t; i < n; i += kPowerThreads) {
    V3 B = v3(bp[i], bp[n + i], bp[2 * n + i]), AC = v3(ap[i], ap[n + i], ap[2 * n + i]);
    tp += (mag2(AC) - mag2(cross(B, AC))) * dt;
  }
  sum[t] = tp;
  __syncthreads();
  for (int w = kPowerThreads / 2; w > 0; w >>= 1) {
    if (t < w) sum[t] += sum[t + w];
    __syncthreads();
  }
  if (t == 0) out[p] = sum[0] * (fabs(qi) * pow(gamma[p], 6.0) / (6 * kPi * kEps0 * kC));
}

// The Lienard-Wiechert field of the trajectory point i at the observer and its arrival time
// (OSCARSSR::CalculateElectricFieldTimeDomain, OSCARSSR.cc:2646-2690; Duke, Synchrotron Radiation, p74):
//   E = q/(4 pi eps0) (1/(1 - n.beta))^3 [ (1 - beta^2)(n - beta)/R^2 + (1/c) n x ((n - beta) x a/c)/R ],
//   t = i dt + R/c, in the reference's vector operation order.
__global__ void efield_time_kernel(const double *__restrict__ X, const double *__restrict__ Bt,
                                   const double *__restrict__ A, int64_t n, double dt, V3 obs, double C0,
                                   double *__restrict__ out_t, double *__restrict__ out_e) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V3 x = v3(X[i], X[n + i], X[2 * n + i]);
  const V3 b = v3(Bt[i], Bt[n + i], Bt[2 * n + i]);
  const V3 ac = v3(A[i], A[n + i], A[2 * n + i]);
  const V3 R = obs - x;
  const double Rm = mag(R);
  const V3 N = R / Rm;  // TVector3D::UnitVector
  const double D = Rm;
  const double Mult = C0 * pow(1.0 / (1.0 - dot(N, b)), 3.0);
  const V3 nb = N - b;
  const double s1 = 1.0 - mag2(b);
  const V3 near = v3(s1 * nb.x, s1 * nb.y, s1 * nb.z) / mag2(R);
  const V3 c = cross(N, cross(nb, ac));
  const double ic = 1.0 / kC;
  const V3 far = v3(ic * c.x, ic * c.y, ic * c.z) / mag(R);
  const V3 sum = near + far;
  out_e[3 * i] = Mult * sum.x;
  out_e[3 * i + 1] = Mult * sum.y;
  out_e[3 * i + 2] = Mult * sum.z;
  out_t[i] = (double)i * dt + D / kC;
}

// Kahan accumulation over particles in order: T3DScalarContainer::AddToPoint (T3DScalarContainer.cc:31-47)
__global__ void accumulate_kernel(const double *__restrict__ vals, int nparticles, int64_t nout, double w,
                                  double *__restrict__ out, double *__restrict__ comp) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nout) return;
  double sum = out[j], c = comp[j];
  for (int p = 0; p < nparticles; ++p) {
    const double v = vals[(int64_t)p * nout + j] * w;
    const double y = v - c, t = sum + y;
    c = (t - sum) - y;
    sum = t;
  }
  out[j] = sum;
  comp[j] = c;
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ---------------------------------------------------------------- launchers

static int64_t tiles_of(int64_t nout, int nparticles) { return (nout + kTile - 1) / kTile * nparticles; }
static int64_t splits(int64_t n, int64_t chunk) { return (n + chunk - 1) / chunk; }
static int64_t flux_chunk(int64_t n, int64_t np, int nparticles) {
  return chunk_for(tiles_of(np, nparticles), n, wave_slots(flux_fp64_kernel, kTile));
}
static int64_t spectrum_chunk(int64_t n, int64_t ne, int nparticles) {
  return chunk_for(tiles_of(ne, nparticles), n, wave_slots(spectrum_fp64_kernel, kTile));
}
static int64_t pd_chunk(int64_t n, int64_t np, int nparticles) {
  return chunk_for(tiles_of(np, nparticles), n, wave_slots(pd_fp64_kernel, kTile));
}

size_t fp64_flux_scratch_bytes(int64_t n, int64_t np, int nparticles) {
  return sizeof(double) * 6 * (size_t)np * nparticles * splits(n, flux_chunk(n, np, nparticles));
}

cudaError_t fp64_flux(const srs_traj_view &t, const srs_beam_consts &b, const double *d_points, int64_t np,
                      double energy_ev, double *d_out, void *scratch, cudaStream_t s) {
  if (np <= 0 || t.nparticles <= 0) return cudaSuccess;
  const int64_t chunk = flux_chunk(t.n, np, t.nparticles);
  const int S = (int)splits(t.n, chunk);
  const double omega = ev_to_omega(energy_ev);
  double *partial = static_cast<double *>(scratch);
  dim3 grid((unsigned)((np + kTile - 1) / kTile), S, t.nparticles);
  if (cudaError_t e = launch_after(flux_fp64_kernel, grid, dim3(kTile), 0, s, t.x, t.beta, t.n, t.dt, d_points, np,
                                   omega, chunk, partial))
    return e;
  return finish_flux_partials(partial, S, np, t.nparticles, nullptr, omega, t.dt, flux_c0(b.charge),
                              flux_c2(b.charge, b.current), d_out, s);
}

size_t fp64_spectrum_scratch_bytes(int64_t n, int64_t ne, int nparticles) {
  return sizeof(double) * 6 * (size_t)ne * nparticles * splits(n, spectrum_chunk(n, ne, nparticles));
}

cudaError_t fp64_spectrum(const srs_traj_view &t, const srs_beam_consts &b, const double obs[3],
                          const double *d_energies, int64_t ne, double *d_out, void *scratch, cudaStream_t s,
                          double *d_e6) {
  if (ne <= 0 || t.nparticles <= 0) return cudaSuccess;
  const int64_t chunk = spectrum_chunk(t.n, ne, t.nparticles);
  const int S = (int)splits(t.n, chunk);
  double *partial = static_cast<double *>(scratch);
  dim3 grid((unsigned)((ne + kTile - 1) / kTile), S, t.nparticles);
  if (cudaError_t e = launch_after(spectrum_fp64_kernel, grid, dim3(kTile), 0, s, t.x, t.beta, t.n, t.dt,
                                   v3(obs[0], obs[1], obs[2]), d_energies, ne, chunk, partial))
    return e;
  return finish_flux_partials(partial, S, ne, t.nparticles, nullptr, 0.0, t.dt, flux_c0(b.charge),
                              flux_c2(b.charge, b.current), d_out, s, d_e6, d_energies);
}

size_t fp64_pd_scratch_bytes(int64_t n, int64_t np, int nparticles) {
  return sizeof(double) * (size_t)np * nparticles * splits(n, pd_chunk(n, np, nparticles));
}

cudaError_t fp64_power_density(const srs_traj_view &t, const srs_beam_consts &b, const double *d_points,
                               const double *d_normals, int64_t np, int directional, double *d_out, void *scratch,
                               cudaStream_t s) {
  if (np <= 0 || t.nparticles <= 0) return cudaSuccess;
  const int64_t chunk = pd_chunk(t.n, np, t.nparticles);
  const int S = (int)splits(t.n, chunk);
  double *partial = static_cast<double *>(scratch);
  dim3 grid((unsigned)((np + kTile - 1) / kTile), S, t.nparticles);
  if (cudaError_t e = launch_after(pd_fp64_kernel, grid, dim3(kTile), 0, s, t.x, t.beta, t.aoc, t.n, d_points,
                                   d_normals, np, directional, chunk, partial))
    return e;
  return finish_pd_partials(partial, S, np, t.nparticles, pd_const(b.charge, b.current) * t.dt, directional, d_out, s);
}

cudaError_t total_power(const srs_traj_view &t, const srs_beam_consts &b, const double *d_gamma, double *d_out,
                        cudaStream_t s) {
  if (t.nparticles <= 0) return cudaSuccess;
  total_power_kernel<<<(unsigned)t.nparticles, kPowerThreads, 0, s>>>(t.beta, t.aoc, t.n, t.dt, b.charge * b.current,
                                                                      d_gamma, d_out);
  return cudaGetLastError();
}

cudaError_t finish_flux_partials(const double *partial, int S, int64_t nout, int nparticles, const double *omegas,
                                 double omega0, double dt, double C0, double C2, double *out, cudaStream_t s,
                                 double *e6, const double *energies) {
  // set up while the sums that wrote the partials finish (the kernel waits for their writes).  Up to 2048
  // outputs 16 groups of chunks, above 4: by then 32 outputs per block fill the GPU, and rows of 32
  // doubles are read in full lines.
  const int64_t total = nout * nparticles;
  if (total <= 2048)
    return launch_after(flux_reduce_kernel<8, 16>, dim3((unsigned)blocks_for(total, 8)), dim3(768), 0, s, partial, S,
                        nout, nparticles, omegas, energies, omega0, dt, C0, C2, out, e6);
  return launch_after(flux_reduce_kernel<32, 4>, dim3((unsigned)blocks_for(total, 32)), dim3(768), 0, s, partial, S,
                      nout, nparticles, omegas, energies, omega0, dt, C0, C2, out, e6);
}

cudaError_t finish_pd_partials(const double *partial, int S, int64_t np, int nparticles, double cdt, int directional,
                               double *out, cudaStream_t s) {
  const int64_t total = np * nparticles;
  if (total <= 4096)
    return launch_after(pd_reduce_kernel<8, 32>, dim3((unsigned)blocks_for(total, 8)), dim3(256), 0, s, partial, S, np,
                        nparticles, cdt, directional, out);
  return launch_after(pd_reduce_kernel<32, 8>, dim3((unsigned)blocks_for(total, 32)), dim3(256), 0, s, partial, S, np,
                      nparticles, cdt, directional, out);
}

cudaError_t accumulate_particles(const double *d_vals, int nparticles, int64_t nout, double weight, double *d_out,
                                 double *d_comp, cudaStream_t s) {
  if (nout <= 0) return cudaSuccess;
  accumulate_kernel<<<blocks_for(nout, 256), 256, 0, s>>>(d_vals, nparticles, nout, weight, d_out, d_comp);
  return cudaGetLastError();
}

cudaError_t efield_time(const srs_traj_view &t, double charge, const double obs[3], double *d_t, double *d_e,
                        cudaStream_t s) {
  if (t.n <= 0) return cudaSuccess;
  const double C0 = charge / (four_pi() * kEps0);  // OSCARSSR.cc:2662
  efield_time_kernel<<<(unsigned)((t.n + 127) / 128), 128, 0, s>>>(t.x, t.beta, t.aoc, t.n, t.dt, ld3(obs), C0, d_t,
                                                                    d_e);
  return cudaGetLastError();
}

}  // namespace srs
