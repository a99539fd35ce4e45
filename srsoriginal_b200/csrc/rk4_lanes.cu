// RK4 trajectories of many particles through ideal undulators along z, one chain of one particle per lane
// (compiled with -fmad=false).
//
// rk4.cu spends a warp's lanes on one particle (fields and stages side by side, shuffles to combine): a
// step costs ~0.87 us there, and a batch is bound by the instructions per particle.  Here one lane
// integrates one chain (forward or backward) of one particle with the step of rk4_und.cuh, bit for bit
// rk4.cu's, bound by the latency of the step (~0.79 us, four sines two by two) whether one lane of the
// warp is used or 16.  So up to 592 x 16 chains take about the time of one, and 592 x 32 twice that; they are spread
// over one warp per scheduler first.  Measured (rk4.cu -> here): 1024 particles of 20001 points 22.0 -> 15.9 ms, 300
// 38.6 -> 15.7 ms, 4096 of 10001 points 12.7 -> 8.4 ms, 18944 of 1001 points 2.9 -> 1.7 ms.  (One double-double sincos per step rotated to the
// other stages took 8.9 ms for 1024, but an ulp in 2 % of the sines flips a last bit of a velocity
// along the flight in some particles, which moves all later phases by ~1e-6 rad: not kept.)
//
// A block is kPairs integrating warps, one per scheduler, and as many storing warps.  An integrating warp
// leaves a step's nine numbers per lane in shared memory (position, velocity, acceleration); every kRing
// / lanes steps its storing warp takes them over, divides by c and writes rows of consecutive points while the next ones are
// computed.  Layout written: [particle][component][point], as rk4.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "rk4_und.cuh"
#include "srs_internal.h"

namespace srs {
namespace {

constexpr int kRing = 256;  // steps x lanes per buffer
constexpr int kPairs = 4;   // of an integrating and a storing warp per block

// Row stride of the ring for L lanes: odd, so that the storing warp's column reads spread over the banks.
__host__ __device__ constexpr int ring_stride(int L) { return L + 1 - (L & 1); }
__host__ __device__ constexpr int ring_doubles(int L) { return kRing / L * 9 * ring_stride(L); }

struct Chain {
  const srs_particle *p;
  double h, *x, *b, *a;
  int64_t n, records, first;  // points per component; states recorded; stored index of state 0
  int dir;
};

// the 64 threads of a pair of warps
__device__ __forceinline__ void pair_barrier(int pair) {
  asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
}

template <int kN>
__global__ void __launch_bounds__(64 * kPairs) rk4_lanes_kernel(const srs_field *__restrict__ gfields, int nfields,
                                                                const srs_particle *__restrict__ particles,
                                                                int nparticles, int chains, double dt_all,
                                                                int64_t nfwd_all, int64_t nbwd_all,
                                                                double *__restrict__ X, double *__restrict__ Bt,
                                                                double *__restrict__ A,
                                                                const TrajSpec *__restrict__ specs, int log2L) {
  extern __shared__ __align__(16) double rings[];  // [pair][2][step][component][lane]
  __shared__ UndField und[kMaxUndulators];
  __shared__ Chain chain[kPairs][32];
  __shared__ long long longest[kPairs];
  const int lane = threadIdx.x & 31, pair = (threadIdx.x >> 5) % kPairs, items = nparticles * chains;
  const bool integrates = threadIdx.x < 32 * kPairs;
  if (threadIdx.x < nfields) prepare_undulator(gfields[threadIdx.x], und[threadIdx.x]);
  const int L = 1 << log2L, steps = kRing >> log2L, ld = ring_stride(L);
  // item -> particle and chain; the backward chain's state 0 is the forward chain's
  auto chain_of = [&](int item) {
    const int p = item / chains, back = item - p * chains;
    Chain c;
    c.p = particles + p;
    const int64_t nf = specs ? specs[p].nfwd : nfwd_all, nb = specs ? specs[p].nbwd : nbwd_all;
    const double dt = specs ? specs[p].dt : dt_all;
    c.n = nf + nb;
    c.x = specs ? specs[p].x : X + (int64_t)p * 3 * c.n;
    c.b = specs ? specs[p].beta : Bt + (int64_t)p * 3 * c.n;
    c.a = specs ? specs[p].aoc : A + (int64_t)p * 3 * c.n;
    c.h = back ? -dt : dt;
    c.records = back ? (nb > 0 ? nb + 1 : 0) : nf;
    c.first = nb;
    c.dir = back ? -1 : 1;
    return c;
  };
  const int item0 = (blockIdx.x * kPairs + pair) * L, mine = item0 + min(lane, L - 1);
  const Chain own = chain_of(min(mine, items - 1));
  if (integrates) {
    long long r = mine < items ? own.records : 0;
    for (int o = 16; o > 0; o >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (lane == 0) longest[pair] = r;
    chain[pair][lane] = own;
  }
  __syncthreads();
  double *const ring = rings + (size_t)pair * 2 * ring_doubles(L);
  UndField held[kN];  // in registers: shared memory would be read again after every store to it
#pragma unroll
  for (int i = 0; i < kN; ++i) held[i] = und[i];
  const double h = own.h, hh = h * 0.5, h6 = h / 6.0, qomg = own.p->qomg, rC = 1.0 / kC;
  V3 pos = ld3(own.p->x0), vel = v3(own.p->beta0[0] * kC, own.p->beta0[1] * kC, own.p->beta0[2] * kC);
  V3 acc = v3(0, 0, 0);
  const int64_t buffers = (longest[pair] + steps - 1) / steps;
  for (int64_t k = 0; k <= buffers; ++k) {
    if (integrates) {
      if (k < buffers) {
        double *o = ring + (k & 1) * ring_doubles(L) + lane;
        for (int s = 0; s < steps; ++s, o += 9 * ld) {
          if (lane < L) {
            o[0] = pos.x; o[ld] = pos.y; o[2 * ld] = pos.z;
            o[3 * ld] = vel.x; o[4 * ld] = vel.y; o[5 * ld] = vel.z;
            o[6 * ld] = acc.x; o[7 * ld] = acc.y; o[8 * ld] = acc.z;
          }
          if (k * steps + s + 1 >= own.records) continue;  // (the phases' bound ends with the chain)
          const Increments d = und_increments<kN>(held, qomg, h, hh, h6, pos, vel);
          pos = v3(pos.x + advance(h6, vel.x, d.r1.x, d.r2.x, d.r3.x), pos.y + advance(h6, vel.y, d.r1.y, d.r2.y, d.r3.y),
                   pos.z + advance(h6, vel.z, d.r1.z, d.r2.z, d.r3.z));
          vel = vel + d.d;
          acc = d.a1;
        }
      }
    } else if (k > 0) {
      const double *const in = ring + ((k - 1) & 1) * ring_doubles(L);
      const int rows = 9 * min(L, items - item0);
      const int64_t rec0 = (k - 1) * steps;
      for (int q = lane; q < rows * steps; q += 32) {
        const int s = q & (steps - 1), row = q / steps, c = row % 9, l = row / 9;
        const Chain &ch = chain[pair][l];
        const int64_t rec = rec0 + s;
        if (rec >= ch.records || (ch.dir < 0 && rec == 0)) continue;
        const double v = in[(s * 9 + c) * ld + l];
        double *const to = (c < 3 ? ch.x : c < 6 ? ch.b : ch.a) + (int64_t)(c % 3) * ch.n + ch.first + ch.dir * rec;
        *to = c < 3 ? v : div_rn(v, kC, rC);
      }
    }
    pair_barrier(pair);
  }
}

template <int kN>
cudaError_t launch(const srs_field *d_fields, int nfields, const srs_particle *d_particles, int nparticles, int chains,
                   double dt, int64_t nfwd, int64_t nbwd, double *d_x, double *d_b, double *d_a, const TrajSpec *d_specs,
                   cudaStream_t s) {
  const int items = nparticles * chains;
  int log2L = 0;
  while (log2L < 5 && (items >> log2L) > 148 * kPairs) ++log2L;  // one integrating warp per scheduler first
  const int L = 1 << log2L, per_block = kPairs * L;
  const size_t smem = sizeof(double) * 2 * kPairs * ring_doubles(L);
  if (cudaError_t e = cudaFuncSetAttribute(rk4_lanes_kernel<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(sizeof(double) * 2 * kPairs * ring_doubles(2))))  // the widest: rows of 3
    return e;
  rk4_lanes_kernel<kN><<<(unsigned)((items + per_block - 1) / per_block), 64 * kPairs, smem, s>>>(
      d_fields, nfields, d_particles, nparticles, chains, dt, nfwd, nbwd, d_x, d_b, d_a, d_specs, log2L);
  return cudaGetLastError();
}

}  // namespace

int undulators_along_z(const srs_field *f, int nfields, const srs_particle *particles, int nparticles, double time,
                       double *reach) {
  if (nfields < 1 || nfields > kMaxUndulators || !finite_starts(particles, nparticles)) return 0;
  double far = kC * time;  // |z| stays below
  for (int p = 0; p < nparticles; ++p) {
    const double *const b = particles[p].beta0;
    if (!(b[0] * b[0] + b[1] * b[1] + b[2] * b[2] <= 1.0 + 1e-9)) return 0;
    far = std::max(far, kC * time + std::fabs(particles[p].x0[2]));
  }
  for (int i = 0; i < nfields; ++i) {
    const double lambda = f[i].period[2];
    if (f[i].kind != SRS_FIELD_UNDULATOR || f[i].taper != 0 || f[i].period[0] != 0 || f[i].period[1] != 0 ||
        !(lambda > 1e-100 && lambda < 1e100) || !(std::fabs(f[i].center[0]) < 1e300) ||
        !(std::fabs(f[i].center[1]) < 1e300))
      return 0;
    // the phases stay below 1e5 rad up to twice that
    if (!((2.0 * far + std::fabs(f[i].center[2])) / lambda + std::fabs(f[i].phase) < 1.5e4)) return 0;
  }
  if (reach) *reach = 1.05 * far;
  return nfields;
}

cudaError_t launch_rk4_lanes(int undulators, const srs_field *d_fields, int nfields, const srs_particle *d_particles,
                             int nparticles, int chains, double dt, int64_t nfwd, int64_t nbwd, double *d_x, double *d_b,
                             double *d_a, const TrajSpec *d_specs, cudaStream_t s) {
  if (nparticles <= 0) return cudaSuccess;
  auto run = [&](auto kernel) {
    return kernel(d_fields, nfields, d_particles, nparticles, chains, dt, nfwd, nbwd, d_x, d_b, d_a, d_specs, s);
  };
  switch (undulators) {
    case 1: return run(launch<1>);
    case 2: return run(launch<2>);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace srs
