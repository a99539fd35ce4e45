// The serial RK4 trajectory, bit for bit, integrated parallel in time (compiled with -fmad=false).
//
// rk4.cu integrates one particle as one chain of ~0.9 us per step (20001 points: 17.3 ms) that no
// width of the GPU shortens: bound by the latency of ~80 dependent FP64 operations, shuffles and a
// sine per step.  Almost all of that work depends on the state only weakly: with the state (p, v) at
// a step's start known approximately, the increments hh*a1, hh*a2, h*a3 and h6*(a1 + a4 + 2(a2 + a3))
// that the step adds to v are known to a relative error of that size, and what remains serial is one
// rounded addition per component and step:
//     v' = RN(v + d),   p' = RN(p + h6*((v + v4) + 2(v3 + v2))),  v2 = RN(v + hh*a1), ...
// So the recurrence is solved by fixed-point (Picard) iteration on the states of all steps:
//
//   pit_pass_kernel    one block per kStepsPerBlock steps: every thread forms its step's increments from
//                      the last iterate, then the block re-adds its steps in order from its start
//                      state.  Every block sums the mismatches that the last iteration left between
//                      the blocks before it and moves its start state by them.  From straight flight
//                      two iterations gain 3-4 digits for ultra-relativistic particles; the components
//                      along the flight direction settle on their exact bits here.
//   pit_steps_kernel   every step's increments from the current states, and the check: the step from
//                      state j, in the serial kernel's arithmetic, must give state j + 1 bit for bit.
//                      If that holds for all steps then, by induction from the exact start state,
//                      the states ARE the serial trajectory.  Also writes the trajectory arrays.
//   pit_chain_kernel   the additions of a whole chain in order (one warp for v, one for p, tile after
//                      tile, the other warps feeding them): one rounded addition, 8 cycles, per step
//                      where the serial kernel needs ~1700.
//
// On long chains (kRunsMinSteps) those additions are spread over the GPU too.  While the sum stays in one
// binade, a rounded addition v + d is the exact addition of d rounded to that binade's grid, whatever v is
// (ties aside), so a run of such steps is one exact addend.  The blocks, which know v nearly, find the runs
// and leave a list of addends (run totals, and the d of the steps in between: a change of binade, a tie):
// 2750 for the x of 20000 steps through an undulator, 625 (one per warp) for y and z.
//
//   pit_starts_kernel  adds a component's list in order, which gives every block's start state;
//   pit_positions_kernel  re-adds the velocities of the blocks from there and lists the positions' runs;
//   then the lists of the positions, and pit_steps_kernel re-adds those.
//
// The lists need no proof: a wrong one (the state known too badly) fails the check and costs a sweep.
//
// Steps and chains alternate until the check holds; the serial kernel runs if it never does (slow
// particles in strong fields, where the iteration does not contract): the result is always the serial
// trajectory, bit for bit.  Both chains of the trajectory (forward from t0, backward) and several
// particles are integrated side by side.
//
// Measured on a B200 around a call (serial kernel -> here): 20001 points through one undulator 17.6 -> 0.20 ms,
// 40001 through two 39.0 -> 0.35 ms, 12001 through a field map in two chains 14.1 -> 0.14 ms, 24 particles of
// 10001 points 9.1 -> 0.44 ms, 2001 points 1.78 -> 0.14 ms, 300 points 0.28 -> 0.11 ms.  A pass is bound by
// latency (~6.5 us: launch, loads, four field evaluations, 2 x 128 additions in order); a sweep takes 0.16 ms
// by the chain kernel on 20001 points, 0.05 ms by runs (20 us per list, 10 us per kernel of blocks).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "rk4_fields.cuh"
#include "rk4_und.cuh"
#include "srs_internal.h"

namespace srs {
namespace {

constexpr int kStepsPerBlock = 128;  // steps (and threads) of a pass block
// Doubles of a component's row in shared memory: the three lanes that add walk on different banks (a third of
// the wavefronts of a pass were these rows' conflicts; 24 particles of 10001 points 560 -> 540 us, 100 of 20001
// 3.46 -> 3.29 ms, where the blocks of several waves share an SM's memory pipe).
constexpr int kRow = kStepsPerBlock + 2;
constexpr int kChainTile = 256;      // steps per tile of the chain kernel
constexpr int kChainThreads = 512;
constexpr int kGroup = 12;           // blocks whose addends the starts kernel holds at a time, one feeding warp each
constexpr int kStartsThreads = 32 * (kGroup + 1);
constexpr int kPasses = 14;          // passes launched (they return at once when the item is ready)
// When an item is given up: the first pass adds up the turns that the fields give on straight flight, and beyond
// kMaxTurn the iteration does not get to the exact bits within the passes and sweeps below; or, where straight
// flight misses the fields, mismatches above kLostMismatch of the speed are left after pass kContracted or a later
// one.  (Lists of undulators along z alone are not summed up: the host knows their strength.)  Measured
// for 300, 2001 and 20001 points in an undulator, a map of one and a map of a dipole: all settle up to a turn of
// 1.0, at 1.2 five of nine, at 1.5 none; after pass 4 at most 9e-3 is left of those that settle.
constexpr double kMaxTurn = 1.3, kLostMismatch = 0.03;
constexpr int kContracted = 4;
constexpr int kSweeps = 4;           // exact sweeps before the serial kernel takes over
// Chains by runs from this length: a sweep of the chain kernel takes 7.8 ns per step of the longest chain
// (1 or 24 particles alike), one by runs ~40 us, 1.5 ns per step and ~20 ns per block of all particles.
// Measured, chain kernel -> runs: 2001 points 128 -> 140 us, 2 x 6000 162 -> 149, 20001 253 -> 172, 40001
// 645 -> 344, 24 particles of 20001 1102 -> 1031, of 10001 556 -> 575, 100 of 20001 3380 -> 3930.
constexpr int64_t kRunsMinSteps = 4500, kRunsStepsPerBlock = 3;

// One chain of one particle.
struct Item {
  int64_t m;       // steps
  int nblk;        // pass blocks
  double h, qomg;
  double s0[6];    // start state: position, velocity
  double *x, *b, *a;
  int64_t n;       // points per component
  int64_t first;   // stored index of state 0 (forward) or of state 1 (backward)
  int dir;         // +1 forward, -1 backward
};

// The trajectories to integrate: common settings, or one spec per particle.
struct Job {
  const srs_particle *particles;
  const TrajSpec *specs;
  double dt;
  int64_t nfwd, nbwd;
  double *x, *b, *a;
  int nparticles, chains;  // chains per particle (2 when some particle has points before t0)
  int64_t stride;          // doubles per component of an item's states
  int maxblk;              // pass blocks of the longest chain
  bool by_runs;            // the chains' additions by runs (kRunsMinSteps)
  double reach, fast2;     // with undulators: bounds on |z| and |v|^2 of all states, which keep the phases below 1e5
};

struct Scratch {
  double *S;      // [item][6][stride]: states
  double *R;      // [item][12][stride]: increments hh*a1, hh*a2, h*a3, d or those of the positions (3 components each)
  double *L;      // [item][3][maxblk][kStepsPerBlock]: addends of a component's chain, block by block
  int *count;     // [item][3][maxblk]: addends of a block
  double *T[2], *E[2];        // [item][maxblk][6]: start state of a block, state after its last step (pass k: k & 1);
                              // T[0] after the passes: the start states that the chains give
  int *ready;                 // per item: the pass that found nothing left to settle, or kPasses
  int *done, *all_ticket;     // the whole job verified; blocks of the steps kernel finished
  unsigned long long *bad;    // steps that do not reproduce (reset by the last block)
  int *failed;                // an item was given up
  float *turn;                // per item: sum |d| of the first pass
  Prepared *prep;
  UndField *und;
  // of pass k.  Selected: an index puts the kernel's argument on the stack of every thread (120 bytes; 24 particles
  // of 10001 points 475 -> 435 us without it, 100 of 5001 770 -> 690, 20001 points 204 -> 202).
  __device__ __forceinline__ double *starts(int k) const { return k & 1 ? T[1] : T[0]; }
  __device__ __forceinline__ double *ends(int k) const { return k & 1 ? E[1] : E[0]; }
};

__device__ inline Item item_of(const Job &J, int it) {
  Item I;
  const int p = it / J.chains, chain = it - p * J.chains;
  const srs_particle &P = J.particles[p];
  int64_t nf = J.nfwd, nb = J.nbwd;
  double dt = J.dt;
  I.n = nf + nb;
  I.x = J.x + (int64_t)p * 3 * I.n;
  I.b = J.b + (int64_t)p * 3 * I.n;
  I.a = J.a + (int64_t)p * 3 * I.n;
  if (J.specs) {
    const TrajSpec &s = J.specs[p];
    nf = s.nfwd;
    nb = s.nbwd;
    dt = s.dt;
    I.n = nf + nb;
    I.x = s.x;
    I.b = s.beta;
    I.a = s.aoc;
  }
  I.m = chain == 0 ? (nf > 0 ? nf - 1 : 0) : nb;
  I.nblk = (int)((I.m + kStepsPerBlock - 1) / kStepsPerBlock);
  I.h = chain == 0 ? dt : -dt;
  I.qomg = P.qomg;
  for (int c = 0; c < 3; ++c) {
    I.s0[c] = P.x0[c];
    I.s0[3 + c] = P.beta0[c] * kC;
  }
  I.first = chain == 0 ? nb : nb - 1;
  I.dir = chain == 0 ? 1 : -1;
  return I;
}

// One copy of the field code: a step evaluates it four times, and a cold instruction cache costs a pass
// more than the calls.
__device__ __noinline__ V3 field_total(const Prepared *sp, const srs_field *sf, int nfields, V3 x) {
  V3 s = v3(0, 0, 0);
  for (int f = 0; f < nfields; ++f) s = s + field_along(sp[f], sf[f], x);
  return s;
}

// The increments of one serial RK4 step that depend on the state only weakly (OSCARSSR.cc:826-874; the
// operations and their order are those of rk4.cu): r1 = hh*a1, r2 = hh*a2, r3 = h*a3,
// d = h6*(a1 + a4 + 2(a3 + a2)).
__device__ __forceinline__ Increments increments(const Prepared *sp, const srs_field *sf, int nfields, double qomg,
                                                 double h, double hh, double h6, V3 pos, V3 vel) {
  auto B = [&](V3 x) { return field_total(sp, sf, nfields, x); };
  Increments o;
  o.a1 = force(qomg, vel, B(pos));
  o.r1 = scale3(hh, o.a1);
  const V3 v2 = vel + o.r1;
  const V3 a2 = force(qomg, v2, B(vadd_scaled(pos, hh, vel)));
  o.r2 = scale3(hh, a2);
  const V3 v3_ = vel + o.r2;
  const V3 a3 = force(qomg, v3_, B(vadd_scaled(pos, hh, v2)));
  o.r3 = scale3(h, a3);
  const V3 v4 = vel + o.r3;
  const V3 a4 = force(qomg, v4, B(vadd_scaled(pos, h, v3_)));
  const V3 m = a3 + a2;
  o.d = v3(h6 * (o.a1.x + a4.x + 2.0 * m.x), h6 * (o.a1.y + a4.y + 2.0 * m.y), h6 * (o.a1.z + a4.z + 2.0 * m.z));
  return o;
}

// The fields of a job as the blocks' threads evaluate them: kN undulators along z, or any list (kN = 0).
template <int kN>
struct Fields {
  UndField und[kMaxUndulators];
  __device__ __forceinline__ void load(const srs_field *, const Scratch &W, int) {
    const long long *a = reinterpret_cast<const long long *>(W.und);
    long long *b = reinterpret_cast<long long *>(und);
    for (int k = threadIdx.x; k < kN * (int)(sizeof(UndField) / 8); k += blockDim.x) b[k] = a[k];
  }
  // An iterate may lie anywhere, or be no number, where a trajectory's state does not: one out of the bounds is not
  // stepped, and fails the check.
  __device__ __forceinline__ Increments step(int, const Job &J, double qomg, double h, double hh, double h6, V3 pos,
                                             V3 vel) const {
    if (!(fabs(pos.z) < J.reach) || !(mag2(vel) < J.fast2)) pos.z = vel.x = vel.y = vel.z = 0.0;
    return und_increments<kN>(und, qomg, h, hh, h6, pos, vel);
  }
};
template <>
struct Fields<0> {
  srs_field sf[kMaxFieldsShared];
  Prepared sp[kMaxFieldsShared];
  __device__ __forceinline__ void load(const srs_field *gf, const Scratch &W, int nfields) {
    copy_fields(sf, sp, gf, W.prep, nfields);
  }
  __device__ __forceinline__ Increments step(int nfields, const Job &, double qomg, double h, double hh, double h6, V3 pos,
                                             V3 vel) const {
    return increments(sp, sf, nfields, qomg, h, hh, h6, pos, vel);
  }
};

// o[j] (which may be d[j]) = the running sum before d[j] is added, for n (a multiple of 16) rounded additions in order; returns
// the sum.  The next sixteen terms are loaded while the current ones are added, so a step costs the
// latency of its addition; a 16-byte access covers two steps.
__device__ __forceinline__ double add_in_order(double acc, const double *d, double *o, int n) {
  double2 nx[8];
  const double2 *const d2 = reinterpret_cast<const double2 *>(d);
  double2 *const o2 = reinterpret_cast<double2 *>(o);
#pragma unroll
  for (int k = 0; k < 8; ++k) nx[k] = d2[k];
  for (int j = 0; j < n / 2; j += 8) {
    double2 cu[8];
    const int jn = j + 8 < n / 2 ? j + 8 : j;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      cu[k] = nx[k];
      nx[k] = d2[jn + k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double2 v;
      v.x = acc;
      acc += cu[k].x;
      v.y = acc;
      acc += cu[k].y;
      o2[j + k] = v;
    }
  }
  return acc;
}

// Whether the rounded addition a + d is the exact addition of r, for every a' in place of a that differs by
// less than tol: a' and a' + d lie in one binade, so the sum is rounded on that binade's grid, which a' is
// on (a tie goes to the even neighbour, which depends on a').
__device__ __forceinline__ bool exact_addend(double a, double d, double tol, double &r) {
  const double s = a + d;
  r = s - a;
  if (d == 0.0) {
    r = d;
    return true;
  }
  const double lo = __longlong_as_double(__double_as_longlong(a) & 0x7ff0000000000000ll), hi = 2.0 * lo;
  const bool same_sign = (__double_as_longlong(a) ^ __double_as_longlong(s)) >= 0;
  return same_sign && fabs(a) >= lo + tol && fabs(a) <= hi - tol && fabs(s) >= lo + tol && fabs(s) <= hi - tol &&
         fabs(d - r) != lo * 0x1p-53;
}

// The addends of a block's additions a + d: a run of steps whose additions are exact on one grid is one
// addend, their sum (exact in any order: the partial sums are differences of numbers of one binade).
__device__ __forceinline__ void emit_addends(const Job &J, const Scratch &W, int it, int s, bool active, V3 a, V3 d,
                                             double tol, int (*counts)[3]) {
  constexpr int kWarps = kStepsPerBlock / 32;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const double av[3] = {a.x, a.y, a.z}, dv[3] = {d.x, d.y, d.z};
  double val[3];
  unsigned heads[3];
  int first[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double r;
    const bool run = !active || exact_addend(av[c], dv[c], tol, r);
    val[c] = !active ? -0.0 : run ? r : dv[c];  // x + -0.0 is x for every x
    const unsigned runs = __ballot_sync(0xffffffffu, run);
    heads[c] = ~(runs & (runs << 1));  // a step that no run continues into
    first[c] = 31 - __clz(heads[c] & (0xffffffffu >> (31 - lane)));
  }
#pragma unroll
  for (int o = 1; o < 32; o *= 2)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double y = __shfl_up_sync(0xffffffffu, val[c], o);
      if (lane - o >= first[c]) val[c] += y;
    }
  if (lane < 3) counts[warp][lane] = __popc(lane == 0 ? heads[0] : lane == 1 ? heads[1] : heads[2]);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int64_t row = ((int64_t)it * 3 + c) * J.maxblk + s;
    int at = 0, all = 0;
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) at += counts[w][c];
      all += counts[w][c];
    }
    if (t == 0) W.count[row] = all;
    if (lane == 31 || (heads[c] >> (lane + 1) & 1))
      W.L[row * kStepsPerBlock + at + __popc(heads[c] & (0xffffffffu >> (31 - lane))) - 1] = val[c];
  }
}

// Bounds on the distance of an approximate state from the exact one, as exact_addend takes them: a wrong
// one costs a sweep, the check decides.
__device__ __forceinline__ double speed_tolerance(const Item &I) { return 0x1p-43 * sqrt(mag2(ld3(I.s0 + 3))); }
__device__ __forceinline__ double position_tolerance(const Item &I) {
  return speed_tolerance(I) * fabs(I.h) * (double)I.m;
}

__global__ void pit_init_kernel(Job J, Scratch W, const srs_field *__restrict__ fields, int nfields, int undulators) {
  allow_next_grid();
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int items = J.nparticles * J.chains;
  if (g < nfields && undulators) prepare_undulator(fields[g], W.und[g]);
  else if (g < nfields) prepare(fields[g], W.prep[g], true);
  if (g == 0) {
    *W.done = 0;
    *W.all_ticket = 0;
    *W.bad = 0;
    *W.failed = 0;
  }
  if (g < items) {
    W.ready[g] = kPasses;
    W.turn[g] = 0.0f;
  }
  if (g >= (int64_t)items * J.maxblk) return;
  const int it = (int)(g / J.maxblk), s = (int)(g - (int64_t)it * J.maxblk);
  const Item I = item_of(J, it);
  const double t = I.h * (double)((int64_t)s * kStepsPerBlock);
  for (int c = 0; c < 3; ++c) {  // straight flight (the first pass starts from T[1])
    W.T[1][6 * g + c] = s == 0 ? I.s0[c] : I.s0[c] + I.s0[3 + c] * t;
    W.T[1][6 * g + 3 + c] = I.s0[3 + c];
  }
}

// The mismatches that pass k left between the blocks of an item, summed over the blocks before block s:
// shift[0..2] of its start position, shift[3..5] of its start velocity (a velocity shift moves the
// positions of all later blocks).  Every thread gets them; returns whether the item has settled: the
// transverse mismatches at the rounding of the speed and none in a component that carries the flight
// (its bits decide the phases); lost: one that this thread looked at is above kLostMismatch.
__device__ inline bool mismatches(const Job &J, const Scratch &W, const Item &I, int it, int s, int k,
                                  double (*red)[kStepsPerBlock / 32], double shift[6], bool *lost) {
  const double *const T = W.starts(k) + 6 * (int64_t)it * J.maxblk, *const E = W.ends(k) + 6 * (int64_t)it * J.maxblk;
  const double v2 = mag2(ld3(I.s0 + 3)), hb = I.h * (double)kStepsPerBlock;
  double sum[6] = {0, 0, 0, 0, 0, 0}, big2 = 0.0;
  int open = 0;
  for (int q = threadIdx.x; q < I.nblk - 1; q += kStepsPerBlock) {
    double t6[6], e6[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      e6[c] = E[6 * q + c];
      t6[c] = T[6 * (q + 1) + c];
    }
    const double left = hb * (double)(s - 1 - q);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double dx = e6[c] - t6[c], dv = e6[3 + c] - t6[3 + c];
      if (q < s) {
        sum[c] += dx + dv * left;
        sum[3 + c] += dv;
      }
      big2 = fmax(big2, dv * dv);
      if ((t6[3 + c] * t6[3 + c] > 0.00390625 * v2 && (dv != 0.0 || dx != 0.0)) || !(dv == dv) || !(dx == dx)) open = 1;
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum[c] += __shfl_xor_sync(0xffffffffu, sum[c], o);
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 6; ++c) red[c][threadIdx.x >> 5] = sum[c];
  const int any = __syncthreads_or(open || big2 > 1e-32 * v2);
  for (int c = 0; c < 6; ++c) {
    shift[c] = 0.0;
    for (int w = 0; w < kStepsPerBlock / 32; ++w) shift[c] += red[c][w];
  }
  *lost = k >= kContracted && big2 > kLostMismatch * kLostMismatch * v2;
  return !any;
}

// Picard iteration number `pass` (see the file comment); in the first the states are straight flight.
template <int kN>
__global__ void __launch_bounds__(kStepsPerBlock) pit_pass_kernel(const srs_field *__restrict__ gfields, int nfields,
                                                                  Job J, Scratch W, int pass) {
  __shared__ Fields<kN> fields;
  __shared__ __align__(16) double sd[3][kRow], sv[3][kRow];
  __shared__ double red[6][kStepsPerBlock / 32];
  wait_for_previous_grid();
  allow_next_grid();
  const int it = blockIdx.y, s = blockIdx.x, t = threadIdx.x;
  // as the passes before this one left it (in this pass other blocks may be writing ready = pass - 1, and all
  // threads of a block have to decide alike)
  const bool settled = W.ready[it] + 1 < pass;
  const float turn = kN == 0 && pass == 1 ? W.turn[it] : 0.0f;
  const Item I = item_of(J, it);
  const int64_t blk = (int64_t)it * J.maxblk + s, i = (int64_t)s * kStepsPerBlock + t;
  fields.load(gfields, W, nfields);
  double *const S = W.S + (int64_t)it * 6 * J.stride;
  double *const T = W.starts(pass) + 6 * blk, *const E = W.ends(pass) + 6 * blk;
  const double h = I.h, hh = h * 0.5, h6 = h / 6.0;
  const bool active = i < I.m;
  V3 vel = ld3(I.s0 + 3), pos = ld3(I.s0) + vel * (h * (double)i);
  if (pass > 0 && active) {
    vel = v3(S[3 * J.stride + i], S[4 * J.stride + i], S[5 * J.stride + i]);
    pos = v3(S[i], S[J.stride + i], S[2 * J.stride + i]);
  }
  double start[6];
  for (int c = 0; c < 6; ++c) start[c] = s < I.nblk ? W.starts(pass + 1)[6 * blk + c] : 0.0;
  if (settled || s >= I.nblk) return;
  if (pass > 0) {
    double shift[6];
    bool lost;
    const bool ready = mismatches(J, W, I, it, s, pass - 1, red, shift, &lost);
    const bool turned = kN == 0 && turn > (float)kMaxTurn * sqrtf((float)mag2(ld3(I.s0 + 3)));
    if (lost || (turned && t == 0)) {
      // all items go to the serial kernel: no further pass of any (one that has settled keeps its number, which
      // its blocks are reading)
      for (int q = 0; q < (int)gridDim.y; ++q)
        if (W.ready[q] == kPasses) W.ready[q] = pass - 1;
      *W.failed = 1;
    }
    if (turned) return;
    if (ready) {
      if (t == 0) W.ready[it] = pass - 1;
      return;
    }
    const V3 dv = ld3(shift + 3);
    vel = vel + dv;
    pos = pos + ld3(shift) + dv * (h * (double)t);
    for (int c = 0; c < 6; ++c) start[c] += shift[c];
  }
#pragma unroll
  for (int c = 0; c < 6; ++c)
    if (t == c) T[c] = start[c];
  __syncthreads();
  Increments o;
  o.d = v3(0, 0, 0);
  if (active) o = fields.step(nfields, J, I.qomg, h, hh, h6, pos, vel);
  if (kN == 0 && pass == 0) {  // (its order does not matter: it decides how the same bits are reached)
    float turn = sqrtf((float)mag2(o.d));
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) turn += __shfl_xor_sync(0xffffffffu, turn, k);
    if ((t & 31) == 0) red[0][t >> 5] = turn;
  }
  sd[0][t] = o.d.x;
  sd[1][t] = o.d.y;
  sd[2][t] = o.d.z;
  __syncthreads();
  if (kN == 0 && pass == 0 && t == kStepsPerBlock - 1)
    atomicAdd(W.turn + it, (float)(red[0][0] + red[0][1] + red[0][2] + red[0][3]));
  // the block's steps in order from its start state: velocities, then positions (three lanes)
  if (t < 3) E[3 + t] = add_in_order(t == 0 ? start[3] : t == 1 ? start[4] : start[5], sd[t], sv[t], kStepsPerBlock);
  __syncthreads();
  vel = v3(sv[0][t], sv[1][t], sv[2][t]);
  sd[0][t] = active ? advance(h6, vel.x, o.r1.x, o.r2.x, o.r3.x) : 0.0;
  sd[1][t] = active ? advance(h6, vel.y, o.r1.y, o.r2.y, o.r3.y) : 0.0;
  sd[2][t] = active ? advance(h6, vel.z, o.r1.z, o.r2.z, o.r3.z) : 0.0;
  __syncthreads();
  if (t < 3) E[t] = add_in_order(t == 0 ? start[0] : t == 1 ? start[1] : start[2], sd[t], sv[t], kStepsPerBlock);
  __syncthreads();
  if (active) {
    S[i] = sv[0][t];
    S[J.stride + i] = sv[1][t];
    S[2 * J.stride + i] = sv[2][t];
    S[3 * J.stride + i] = vel.x;
    S[4 * J.stride + i] = vel.y;
    S[5 * J.stride + i] = vel.z;
  }
}

// Every step's increments from the current states, the check, the trajectory arrays, and the addends of the
// velocities' chain (see the file comment).  from_passes: the states are the last pass's and still have
// to be moved by its shifts; otherwise the positions follow from their chain and their increments.
template <int kN, bool kRuns>
__global__ void __launch_bounds__(kStepsPerBlock) pit_steps_kernel(const srs_field *__restrict__ gfields, int nfields,
                                                                   Job J, Scratch W, int from_passes) {
  __shared__ Fields<kN> fields;
  __shared__ __align__(16) double sd[3][kRuns ? kRow : 2], sx[3][kRuns ? kRow : 2];
  __shared__ double red[6][kStepsPerBlock / 32];
  __shared__ int counts[kStepsPerBlock / 32][3];
  wait_for_previous_grid();
  allow_next_grid();
  if (*W.done || *W.failed) return;
  const int it = blockIdx.y, s = blockIdx.x, t = threadIdx.x;
  const Item I = item_of(J, it);
  fields.load(gfields, W, nfields);
  const int64_t i = (int64_t)s * kStepsPerBlock + t;
  double *const S = W.S + (int64_t)it * 6 * J.stride, *const R = W.R + (int64_t)it * 12 * J.stride + i;
  V3 pos = v3(0, 0, 0), vel = v3(0, 0, 0), nv = v3(0, 0, 0);
  if (i < I.m) {
    vel = v3(S[3 * J.stride + i], S[4 * J.stride + i], S[5 * J.stride + i]);
    if (from_passes || !kRuns) pos = v3(S[i], S[J.stride + i], S[2 * J.stride + i]);
    if (kRuns && !from_passes) nv = v3(S[3 * J.stride + i + 1], S[4 * J.stride + i + 1], S[5 * J.stride + i + 1]);
  }
  if (s < I.nblk) {
    if (from_passes) {
      double shift[6];
      bool lost;  // the passes return at once after the one that found the item settled
      mismatches(J, W, I, it, s, min(W.ready[it], kPasses - 1), red, shift, &lost);
      const V3 dv = ld3(shift + 3);
      vel = vel + dv;
      pos = pos + ld3(shift) + dv * (I.h * (double)t);
    } else if constexpr (kRuns) {
      const double *const at = W.T[0] + 6 * ((int64_t)it * J.maxblk + s);
#pragma unroll
      for (int c = 0; c < 3; ++c) sd[c][t] = i < I.m ? R[(9 + c) * J.stride] : 0.0;
      __syncthreads();
      if (t < 3) {
        const double end = add_in_order(at[t], sd[t], sx[t], kStepsPerBlock);
        sx[t][kStepsPerBlock] = s + 1 < I.nblk ? at[6 + t] : end;
      }
      __syncthreads();
      pos = v3(sx[0][t], sx[1][t], sx[2][t]);
    }
  }
  __syncthreads();
  const double rC = 1.0 / kC;
  auto store = [&](int64_t k, V3 p, V3 v, V3 a) {
    I.x[k] = p.x; I.x[I.n + k] = p.y; I.x[2 * I.n + k] = p.z;
    I.b[k] = div_rn(v.x, kC, rC); I.b[I.n + k] = div_rn(v.y, kC, rC); I.b[2 * I.n + k] = div_rn(v.z, kC, rC);
    I.a[k] = div_rn(a.x, kC, rC); I.a[I.n + k] = div_rn(a.y, kC, rC); I.a[2 * I.n + k] = div_rn(a.z, kC, rC);
  };
  int bad = 0;
  if (i == 0 && I.dir > 0 && I.n > I.first) store(I.first, ld3(I.s0), ld3(I.s0 + 3), v3(0, 0, 0));
  Increments o;
  o.d = v3(0, 0, 0);
  if (i < I.m) {
    if (kRuns) {
      S[i] = pos.x;
      S[J.stride + i] = pos.y;
      S[2 * J.stride + i] = pos.z;
    }
    const double hh = I.h * 0.5, h6 = I.h / 6.0;
    o = fields.step(nfields, J, I.qomg, I.h, hh, h6, pos, vel);
    const V3 *const part[4] = {&o.r1, &o.r2, &o.r3, &o.d};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      R[(3 * q) * J.stride] = part[q]->x;
      R[(3 * q + 1) * J.stride] = part[q]->y;
      R[(3 * q + 2) * J.stride] = part[q]->z;
    }
    if (from_passes) {
      bad = 1;  // moved by approximate shifts: to be re-added in order first
    } else {
      if (!kRuns) nv = v3(S[3 * J.stride + i + 1], S[4 * J.stride + i + 1], S[5 * J.stride + i + 1]);
      const V3 np_ = kRuns ? v3(sx[0][t + 1], sx[1][t + 1], sx[2][t + 1])
                               : v3(S[i + 1], S[J.stride + i + 1], S[2 * J.stride + i + 1]);
      auto same = [](double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); };
      bad = !(same(nv.x, vel.x + o.d.x) && same(nv.y, vel.y + o.d.y) && same(nv.z, vel.z + o.d.z) &&
              same(np_.x, pos.x + advance(h6, vel.x, o.r1.x, o.r2.x, o.r3.x)) &&
              same(np_.y, pos.y + advance(h6, vel.y, o.r1.y, o.r2.y, o.r3.y)) &&
              same(np_.z, pos.z + advance(h6, vel.z, o.r1.z, o.r2.z, o.r3.z)));
      store(I.first + I.dir * (I.dir > 0 ? i + 1 : i), np_, nv, o.a1);
    }
  }
  if constexpr (kRuns)
    if (s < I.nblk) emit_addends(J, W, it, s, i < I.m, vel, o.d, speed_tolerance(I), counts);
  bad = __syncthreads_count(bad);
  if (t == 0) {
    if (bad) atomicAdd(W.bad, (unsigned long long)bad);
    __threadfence();
    if (atomicAdd(W.all_ticket, 1) == (int)(gridDim.x * gridDim.y) - 1) {
      __threadfence();
      const unsigned long long total = atomicAdd(W.bad, 0ull);
      *W.bad = 0;
      *W.all_ticket = 0;
      *W.done = total == 0;
    }
  }
}

// The additions of one chain in order, tile after tile: warp 0 (three lanes) the velocities of tile k,
// warp 1 the positions of tile k - 2, the other warps the position increments of tile k - 1, the loads
// of tile k + 1 and the stores.  Bound by the latency of one FP64 addition (8 cycles) per step.
__global__ void __launch_bounds__(kChainThreads) pit_chain_kernel(Job J, Scratch W) {
  __shared__ __align__(16) double sd[2][3][kChainTile], sv[2][3][kChainTile], se[2][3][kChainTile],
      sx[2][3][kChainTile];
  wait_for_previous_grid();
  allow_next_grid();
  if (*W.done || *W.failed) return;
  const int it = blockIdx.x, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const Item I = item_of(J, it);
  if (I.m == 0) return;
  double *const S = W.S + (int64_t)it * 6 * J.stride;
  const double *const R = W.R + (int64_t)it * 12 * J.stride;
  const int64_t tiles = I.m / kChainTile + 1;  // of the m + 1 states
  const double h6 = I.h / 6.0;
  // the feeding warps are those of the two schedulers that the adding warps 0 and 1 are not on
  const bool feeds = (warp & 2) != 0;
  constexpr int kFeeders = kChainThreads / 2, kEach = 3 * kChainTile / kFeeders;
  static_assert(kEach * kFeeders == 3 * kChainTile, "the feeders share a tile evenly");
  const int ft = ((warp >> 2) * 2 + (warp & 1)) * 32 + lane;
  auto load = [&](int64_t k) {  // the increments d of tile k (none after the last state)
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
      const int e = ft + q * kFeeders, c = e / kChainTile, j = e % kChainTile;
      const int64_t g = k * kChainTile + j;
      sd[k & 1][c][j] = g < I.m ? R[(9 + c) * J.stride + g] : 0.0;
    }
  };
  if (feeds) load(0);
  double acc = lane < 3 ? (warp == 0 ? I.s0[3 + lane] : I.s0[lane]) : 0.0;
  __syncthreads();
  for (int64_t k = 0; k < tiles + 3; ++k) {
    if (warp == 0) {
      if (k < tiles && lane < 3) acc = add_in_order(acc, sd[k & 1][lane], sv[k & 1][lane], kChainTile);
    } else if (warp == 1) {
      const int64_t kk = k - 2;
      if (kk >= 0 && kk < tiles && lane < 3) acc = add_in_order(acc, se[kk & 1][lane], sx[kk & 1][lane], kChainTile);
    } else if (feeds) {
      const int64_t kv = k - 1, kx = k - 3;
      if (kv >= 0 && kv < tiles) {
        double r[kEach][3];
#pragma unroll
        for (int q = 0; q < kEach; ++q) {
          const int e = ft + q * kFeeders, c = e / kChainTile;
          const int64_t g = kv * kChainTile + e % kChainTile;
          for (int u = 0; u < 3; ++u) r[q][u] = g < I.m ? R[(3 * u + c) * J.stride + g] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kEach; ++q) {
          const int e = ft + q * kFeeders, c = e / kChainTile, j = e % kChainTile;
          const int64_t g = kv * kChainTile + j;
          const double v = sv[kv & 1][c][j];
          se[kv & 1][c][j] = g < I.m ? advance(h6, v, r[q][0], r[q][1], r[q][2]) : 0.0;
          if (g <= I.m) S[(3 + c) * J.stride + g] = v;
        }
      }
      if (k + 1 < tiles) load(k + 1);
      if (kx >= 0 && kx < tiles) {
#pragma unroll
        for (int q = 0; q < kEach; ++q) {
          const int e = ft + q * kFeeders, c = e / kChainTile, j = e % kChainTile;
          const int64_t g = kx * kChainTile + j;
          if (g <= I.m) S[c * J.stride + g] = sx[kx & 1][c][j];
        }
      }
    }
    __syncthreads();
  }
}

// The start states of the blocks: the additions of one component of an item's velocities (first = 3) or
// positions (first = 0) in order.  The last warp adds (one lane), the others feed it: warp w gathers the addends of
// block w of a group and writes its start state when the group is added.
__global__ void __launch_bounds__(kStartsThreads) pit_starts_kernel(Job J, Scratch W, int first) {
  __shared__ __align__(16) double a[3][kGroup * kStepsPerBlock + 16];
  __shared__ int total[3];
  wait_for_previous_grid();
  allow_next_grid();
  if (*W.done || *W.failed) return;
  const int it = blockIdx.y, c = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Item I = item_of(J, it);
  const int groups = (I.nblk + kGroup - 1) / kGroup;
  const int64_t row = ((int64_t)it * 3 + c) * J.maxblk;
  double acc = I.s0[first + c];
  int cn = 0, off[3] = {0, 0, 0};  // counts of a group's blocks; this warp's first addend in the last three groups
  double val[kStepsPerBlock / 32];
  auto counts = [&](int k) { return lane < kGroup && k * kGroup + lane < I.nblk ? W.count[row + k * kGroup + lane] : 0; };
  auto fetch = [&](int k, int n) {  // the n addends of this warp's block of group k
    const double *const L = W.L + (row + (int64_t)k * kGroup + warp) * kStepsPerBlock;
#pragma unroll
    for (int q = 0; q < kStepsPerBlock / 32; ++q) val[q] = lane + 32 * q < n ? L[lane + 32 * q] : 0.0;
  };
  const bool feeds = warp < kGroup;
  int next = 0;
  if (feeds) {
    cn = counts(0);
    next = counts(1);
    fetch(0, __shfl_sync(0xffffffffu, cn, warp));
  }
  for (int k = 0; k < groups + 2; ++k) {  // group k is gathered, group k - 1 added, group k - 2 written
    if (feeds) {
      int sum = cn;
#pragma unroll
      for (int o = 1; o < kGroup; o *= 2) {
        const int y = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += y;
      }
      const int n = __shfl_sync(0xffffffffu, cn, warp), all = __shfl_sync(0xffffffffu, sum, kGroup - 1);
      off[2] = off[1];
      off[1] = off[0];
      off[0] = __shfl_sync(0xffffffffu, sum, warp) - n;
      if (k < groups) {
#pragma unroll
        for (int q = 0; q < kStepsPerBlock / 32; ++q)
          if (lane + 32 * q < n) a[k % 3][off[0] + lane + 32 * q] = val[q];
        if (warp == 0 && lane < 16) a[k % 3][all + lane] = -0.0;  // (adds nothing)
        if (warp == 0 && lane == 0) total[k % 3] = all;
      }
      cn = next;
      fetch(k + 1, __shfl_sync(0xffffffffu, cn, warp));
      next = counts(k + 2);
      const int b = (k - 2) * kGroup + warp;
      if (k >= 2 && b < I.nblk && lane == 0) W.T[0][6 * ((int64_t)it * J.maxblk + b) + first + c] = a[(k - 2) % 3][off[2]];
    } else if (k >= 1 && k <= groups && lane == 0) {
      acc = add_in_order(acc, a[(k - 1) % 3], a[(k - 1) % 3], (total[(k - 1) % 3] + 15) / 16 * 16);
    }
    __syncthreads();
  }
}

// The velocities from their blocks' start states, the increments of the positions, and the addends of
// the positions' chain.
__global__ void __launch_bounds__(kStepsPerBlock) pit_positions_kernel(Job J, Scratch W) {
  __shared__ __align__(16) double sd[3][kRow], sv[3][kRow];
  __shared__ int counts[kStepsPerBlock / 32][3];
  wait_for_previous_grid();
  allow_next_grid();
  if (*W.done || *W.failed) return;
  const int it = blockIdx.y, s = blockIdx.x, t = threadIdx.x;
  const Item I = item_of(J, it);
  if (s >= I.nblk) return;
  const int64_t i = (int64_t)s * kStepsPerBlock + t;
  const bool active = i < I.m;
  double *const S = W.S + (int64_t)it * 6 * J.stride + i, *const R = W.R + (int64_t)it * 12 * J.stride + i;
  V3 r[4], pos = v3(0, 0, 0);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    r[q] = active ? v3(R[3 * q * J.stride], R[(3 * q + 1) * J.stride], R[(3 * q + 2) * J.stride]) : v3(0, 0, 0);
  if (active) pos = v3(S[0], S[J.stride], S[2 * J.stride]);
  sd[0][t] = r[3].x;
  sd[1][t] = r[3].y;
  sd[2][t] = r[3].z;
  __syncthreads();
  if (t < 3) {
    const double end = add_in_order(W.T[0][6 * ((int64_t)it * J.maxblk + s) + 3 + t], sd[t], sv[t], kStepsPerBlock);
    if ((int64_t)(s + 1) * kStepsPerBlock == I.m) W.S[((int64_t)it * 6 + 3 + t) * J.stride + I.m] = end;
  }
  __syncthreads();
  const V3 vel = v3(sv[0][t], sv[1][t], sv[2][t]);
  if (i <= I.m) {
    S[3 * J.stride] = vel.x;
    S[4 * J.stride] = vel.y;
    S[5 * J.stride] = vel.z;
  }
  const double h6 = I.h / 6.0;
  const V3 d = v3(advance(h6, vel.x, r[0].x, r[1].x, r[2].x), advance(h6, vel.y, r[0].y, r[1].y, r[2].y),
                  advance(h6, vel.z, r[0].z, r[1].z, r[2].z));
  if (active) {
    R[9 * J.stride] = d.x;
    R[10 * J.stride] = d.y;
    R[11 * J.stride] = d.z;
  }
  emit_addends(J, W, it, s, active, pos, d, position_tolerance(I), counts);
}

__global__ void route_kernel(int32_t *route, int nparticles, const int *done) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nparticles) route[p] = !done ? SRS_TRAJ_ROUTE_LANES : *done ? SRS_TRAJ_ROUTE_PARALLEL : SRS_TRAJ_ROUTE_GIVEN_UP;
}

Job make_job(const srs_particle *d_particles, const TrajSpec *d_specs, const TrajSpec *h_specs, int nparticles, double dt,
             int64_t nfwd, int64_t nbwd, double *d_x, double *d_b, double *d_a) {
  Job J;
  J.particles = d_particles;
  J.specs = d_specs;
  J.dt = dt;
  J.nfwd = nfwd;
  J.nbwd = nbwd;
  J.x = d_x;
  J.b = d_b;
  J.a = d_a;
  J.nparticles = nparticles;
  int64_t mf = nfwd - 1, mb = nbwd;
  if (h_specs) {
    mf = mb = 0;
    for (int p = 0; p < nparticles; ++p) {
      mf = std::max(mf, h_specs[p].nfwd - 1);
      mb = std::max(mb, h_specs[p].nbwd);
    }
  }
  J.chains = mb > 0 ? 2 : 1;
  const int64_t m = std::max<int64_t>(std::max(mf, mb), 0);
  J.stride = (m + 2) / 2 * 2;
  J.maxblk = (int)((m + kStepsPerBlock - 1) / kStepsPerBlock);
  J.reach = J.fast2 = 0.0;
  J.by_runs = m >= kRunsMinSteps + kRunsStepsPerBlock * J.nparticles * J.chains * J.maxblk;
  return J;
}

size_t carve(const Job &J, int nfields, void *base, Scratch *W) {
  const size_t items = (size_t)J.nparticles * J.chains, blocks = items * (size_t)std::max(1, J.maxblk);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 15) / 16 * 16;
    return static_cast<char *>(base) + o;
  };
  Scratch s;
  s.S = (double *)take(sizeof(double) * 6 * items * J.stride);
  s.R = (double *)take(sizeof(double) * 12 * items * J.stride);
  s.L = (double *)take(J.by_runs ? sizeof(double) * 3 * blocks * kStepsPerBlock : 0);
  s.count = (int *)take(J.by_runs ? sizeof(int) * 3 * blocks : 0);
  for (int k = 0; k < 2; ++k) {
    s.T[k] = (double *)take(sizeof(double) * 6 * blocks);
    s.E[k] = (double *)take(sizeof(double) * 6 * blocks);
  }
  s.ready = (int *)take(sizeof(int) * items);
  s.done = (int *)take(sizeof(int));
  s.all_ticket = (int *)take(sizeof(int));
  s.failed = (int *)take(sizeof(int));
  s.turn = (float *)take(sizeof(float) * items);
  s.bad = (unsigned long long *)take(sizeof(unsigned long long));
  s.prep = (Prepared *)take(sizeof(Prepared) * (size_t)std::max(1, nfields));
  s.und = (UndField *)take(sizeof(UndField) * kMaxUndulators);
  if (W) *W = s;
  return off;
}

}  // namespace

// When the parallel iteration is used: trajectories long enough to pay for its ~30 launches, and few
// enough of them: it costs ~1.7 ns per step and particle, the serial kernels 0.78 us (rk4_lanes.cu) or
// 0.87 us (rk4.cu) per step of up to 592 particles and more, so they meet near 500 particles; its 144
// bytes of scratch per step and particle (0.7 GB for 256 of 20001 points; 168 by runs) end it before.
constexpr int64_t kExactMinSteps = 256;
constexpr int kExactMaxParticles = 256;
// Longer batches go half by half, so that the scratch kept in the library's pool stays bounded (4 GB: 64 particles of
// 430000 points at a time; a pass fills the GPU long before).  One particle takes what it needs, up to 2^26
// steps: every block sums all the mismatches before it, which costs as much as the serial kernel near 10^8
// (4 million points 0.12 s, serially 3.5 s).
constexpr size_t kExactMaxScratch = (size_t)4 << 30;
constexpr int64_t kExactMaxSteps = (int64_t)1 << 26;
// And only where the iteration contracts: the angle by which the fields could turn a particle over the
// whole trajectory, |q/(m gamma)| sum |B| T (grids not counted: their samples are on the device).  3 GeV
// electrons in 1 T over 2 m: 0.2.  Through an undulator at 2.0 300, 2001 and 20001 points settle, at 2.4 two of
// the three do not; other shapes may fill a part of the way only.  What is given up after the first pass costs 55 to
// 80 us before the serial kernel (0.1 GeV through a 1 T map: 300 points 376 -> 458 us, 2001 2335 -> 2391; when all
// passes and sweeps ran for it, 537 and 2518).
constexpr double kExactMaxTurn = 3.0, kExactMaxTurnUndulators = 2.2;

// More particles through undulators go one chain per lane (rk4_lanes.cu), where that is the faster kernel: from 128
// steps (257 to 4096 particles of 20 points 53-66 against 53-76 us, of 2 26-42 against 40-57, of 100 133-181 against
// 114-169), and not just above the counts where its time nearly doubles at once, as the warps' lanes fill beyond 16
// and as a second warp per scheduler begins (1001 points, serial against lanes: 9400 particles 1.44 / 0.97 ms, 9500
// 1.55 / 1.65, 10000 1.77 / 1.66; 18944 2.90 / 1.70, 19000 2.89 / 3.27, 20000 3.33 / 3.28; 60000 8.8 / 6.8; through two
// undulators, and with two chains, only the second).
constexpr int64_t kLanesMinSteps = 128, kSchedulers = 148 * 4;
static bool lanes_pay(int undulators, int64_t items, int chains) {
  auto just_above = [&](int64_t count) { return items > count && items < count + count / 20; };
  return !(undulators == 1 && chains == 1 && just_above(kSchedulers * 16)) && !just_above(kSchedulers * 32);
}

static double turn_bound(const srs_field *fields, int nfields, const srs_particle *particles, int nparticles, double time) {
  double b = 0.0, q = 0.0;
  for (int f = 0; f < nfields; ++f)
    if (field_shape(fields[f].kind) != SRS_FIELD_GRID) b += mag(ld3(fields[f].field));
  for (int p = 0; p < nparticles; ++p) {
    if (std::isnan(particles[p].qomg)) return particles[p].qomg;  // (no bound: std::max would drop it)
    q = std::max(q, fabs(particles[p].qomg));
  }
  return q * b * time;
}

template <int kN>
static cudaError_t launch_exact(const Job &J, const Scratch &W, const srs_field *d_fields, int nfields, dim3 grid,
                                cudaStream_t s) {
  const dim3 block(kStepsPerBlock);
  for (int k = 0; k < kPasses; ++k)
    if (cudaError_t e = launch_after(pit_pass_kernel<kN>, grid, block, 0, s, d_fields, nfields, J, W, k)) return e;
  const auto steps = J.by_runs ? pit_steps_kernel<kN, true> : pit_steps_kernel<kN, false>;
  const dim3 starts(3, grid.y), starts_threads(kStartsThreads);
  for (int k = 0; k <= kSweeps; ++k) {
    if (cudaError_t e = launch_after(steps, grid, block, 0, s, d_fields, nfields, J, W, k == 0 ? 1 : 0)) return e;
    if (k == kSweeps) break;
    if (!J.by_runs) {
      if (cudaError_t e = launch_after(pit_chain_kernel, dim3(grid.y), dim3(kChainThreads), 0, s, J, W)) return e;
      continue;
    }
    if (cudaError_t e = launch_after(pit_starts_kernel, starts, starts_threads, 0, s, J, W, 3)) return e;
    if (cudaError_t e = launch_after(pit_positions_kernel, grid, block, 0, s, J, W)) return e;
    if (cudaError_t e = launch_after(pit_starts_kernel, starts, starts_threads, 0, s, J, W, 0)) return e;
  }
  return cudaGetLastError();
}

cudaError_t launch_trajectories(const srs_field *d_fields, int nfields, const srs_particle *d_particles, int nparticles,
                                double dt, int64_t nfwd, int64_t nbwd, double *d_x, double *d_b, double *d_a,
                                const TrajSpec *d_specs, const TrajSpec *host_specs, cudaStream_t s,
                                const srs_field *host_fields, const srs_particle *host_particles, int32_t *d_route) {
  if (nparticles <= 0) return cudaSuccess;
  if (nfields > kMaxFieldsShared) return cudaErrorInvalidValue;
  auto routed = [&](cudaError_t e, const int *done) {  // (after the launches that it tells about)
    if (e != cudaSuccess || !d_route) return e;
    route_kernel<<<(unsigned)((nparticles + 127) / 128), 128, 0, s>>>(d_route, nparticles, done);
    return cudaGetLastError();
  };
  const int64_t stage_doubles = nfields > 0 ? grid_stage_doubles(host_fields, nfields) : 0;
  const bool electric = has_electric(host_fields, nfields);
  double time = dt * (double)(nfwd + nbwd), step = dt;
  int64_t steps = std::max(nfwd - 1, nbwd);
  if (host_specs)
    for (int p = 0; p < nparticles; ++p) {
      time = std::max(time, host_specs[p].dt * (double)(host_specs[p].nfwd + host_specs[p].nbwd));
      step = std::max(step, host_specs[p].dt);
      steps = std::max({steps, host_specs[p].nfwd - 1, host_specs[p].nbwd});
    }
  Job J = make_job(d_particles, d_specs, host_specs, nparticles, dt, nfwd, nbwd, d_x, d_b, d_a);
  const int64_t items = (int64_t)nparticles * J.chains, padded = (int64_t)J.maxblk * kStepsPerBlock;
  auto serial = [&](const int *d_skip) {
    if (d_route && !d_skip)
      if (cudaError_t e = cudaMemsetAsync(d_route, 0, sizeof(int32_t) * (size_t)nparticles, s)) return e;
    return launch_rk4(d_fields, nfields, d_particles, nparticles, dt, nfwd, nbwd, d_x, d_b, d_a, s, stage_doubles,
                      electric, d_specs, d_skip);
  };
  const bool few = nparticles <= kExactMaxParticles;
  if (electric || (few ? padded <= kExactMinSteps || padded > kExactMaxSteps : steps < kLanesMinSteps))
    return serial(nullptr);
  if (few && !finite_starts(host_particles, nparticles)) return serial(nullptr);
  // The undulators' phases are bounded by the way that the particles can go.  In one field a step of less than 2.8
  // rad does not lengthen the velocity, but its stages may lie in different fields: then v' = (1 + A + ...) v with A
  // antisymmetric, |A| <= t, the step's turn, and further terms of t^2 / 2, t^3 / 6 and t^4 / 24 at most, so |v'| <= |v|
  // (1 + t^2 + ...) < |v| exp(1.2 t^2) for t < 1, and exp(1.2 T t) over all steps of T rad together.
  const double turn = turn_bound(host_fields, nfields, host_particles, nparticles, time);
  const double step_turn = turn_bound(host_fields, nfields, host_particles, nparticles, step);
  const double growth = exp(1.2 * turn * step_turn);
  int undulators = 0;
  if (step_turn < 1.0) undulators = undulators_along_z(host_fields, nfields, host_particles, nparticles, time * growth, &J.reach);
  J.fast2 = 1.05 * kC * kC * growth * growth;
  if (!few) {
    if (!undulators || !lanes_pay(undulators, items, J.chains)) return serial(nullptr);
    return routed(launch_rk4_lanes(undulators, d_fields, nfields, d_particles, nparticles, J.chains, dt, nfwd, nbwd, d_x,
                                   d_b, d_a, d_specs, s),
                  nullptr);
  }
  if (!(turn < (undulators ? kExactMaxTurnUndulators : kExactMaxTurn))) return serial(nullptr);
  const size_t bytes = carve(J, nfields, nullptr, nullptr);
  if (bytes > kExactMaxScratch && nparticles > 1) {
    const int half = nparticles / 2;
    auto part = [&](int p, int count) {
      const int64_t at = d_specs ? 0 : (int64_t)p * 3 * (nfwd + nbwd);  // (specs carry their own arrays)
      return launch_trajectories(d_fields, nfields, d_particles + p, count, dt, nfwd, nbwd, d_x + at, d_b + at, d_a + at,
                                 d_specs ? d_specs + p : nullptr, host_specs ? host_specs + p : nullptr, s, host_fields,
                                 host_particles + p, d_route ? d_route + p : nullptr);
    };
    if (cudaError_t e = part(0, half)) return e;
    return part(half, nparticles - half);
  }
  DeviceBuffer scratch;
  if (scratch.alloc(bytes, s) != cudaSuccess) {
    cudaGetLastError();  // no room for the states: the serial kernels need none
    return serial(nullptr);
  }
  Scratch W;
  carve(J, nfields, scratch.ptr, &W);
  const dim3 grid((unsigned)std::max(1, J.maxblk), (unsigned)items);
  const int64_t init = std::max<int64_t>(items * std::max(1, J.maxblk), nfields);
  pit_init_kernel<<<(unsigned)((init + 127) / 128), 128, 0, s>>>(J, W, d_fields, nfields, undulators);
  const cudaError_t e = undulators == 1   ? launch_exact<1>(J, W, d_fields, nfields, grid, s)
                        : undulators == 2 ? launch_exact<2>(J, W, d_fields, nfields, grid, s)
                                          : launch_exact<0>(J, W, d_fields, nfields, grid, s);
  if (e != cudaSuccess) return e;
  if (cudaError_t e = cudaGetLastError()) return e;
  return routed(serial(W.done), W.done);  // the serial kernel returns at once when the check held
}

}  // namespace srs
