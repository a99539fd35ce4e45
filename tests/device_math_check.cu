// The FP64 sums' own arithmetic on a GPU (run by tests/test_gpu_units.py), compiled as they are: sqrt_both and the
// quotients formed with it bit for bit against CUDA's correctly rounded square root and division, its reciprocal
// root, reciprocal and the sums' sine and cosine against long double on the host.
//   1/sqrt(a): the last fused operation rounds by 2^-53, the remainder's rounding adds half of that: 1.7e-16.
//   1/a: only the last rounding is left after two Newton steps: 1.2e-16.
//   sin, cos: two roundings of the reduced argument (5.6e-17 each), one or two of the result, w's: 2.4e-16 in all
//   below 2^46 rad; beyond, k may be a neighbour's and the polynomials go past pi/4: 4e-16.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "srs_device.cuh"

using namespace srs;

__global__ void roots(const double *in, int n, double *y, double *inv, unsigned long long *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V3 R = ld3(in + 3 * i);
  const double a = mag2(R);
  double m;
  sqrt_both(a, m, y[i]);
  inv[i] = reciprocal(a);
  const bool good = m == __dsqrt_rn(a) && div_rn(R.x, m, y[i]) == __ddiv_rn(R.x, m) &&
                    div_rn(R.y, m, y[i]) == __ddiv_rn(R.y, m) && div_rn(R.z, m, y[i]) == __ddiv_rn(R.z, m);
  if (!good) atomicAdd(bad, 1ull);
}
__global__ void sines(const double *x, int n, double *s, double *c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (phases_far(x[i], 1.0)) sincos_phase<true>(x[i], s[i], c[i]);
  else sincos_phase<false>(x[i], s[i], c[i]);
}

static constexpr int kN = 1 << 20;

struct Buffers {
  double *d[4];
  unsigned long long *bad;
  Buffers() {
    for (auto &p : d) cudaMalloc(&p, sizeof(double) * 3 * kN);
    cudaMalloc(&bad, sizeof *bad);
  }
};

int main() {
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  Buffers B;
  int fail = 0;
  std::vector<double> in(3 * kN), a(kN), b(kN);
  // observers at a screen, near ones, and vectors of 1e-8 to 1e8 m
  for (int kind = 0; kind < 3; ++kind) {
    for (int i = 0; i < kN; ++i)
      for (int c = 0; c < 3; ++c)
        in[3 * i + c] = kind == 0 ? (c < 2 ? 0.05 * U(rng) : 30.0 + U(rng)) : kind == 1 ? 3.0 * U(rng)
                                  : U(rng) * std::pow(10.0, 8.0 * U(rng));
    cudaMemset(B.bad, 0, sizeof *B.bad);
    cudaMemcpy(B.d[0], in.data(), sizeof(double) * 3 * kN, cudaMemcpyHostToDevice);
    roots<<<kN / 128, 128>>>(B.d[0], kN, B.d[1], B.d[2], B.bad);
    unsigned long long bad = 0;
    cudaMemcpy(&bad, B.bad, sizeof bad, cudaMemcpyDeviceToHost);
    cudaMemcpy(a.data(), B.d[1], sizeof(double) * kN, cudaMemcpyDeviceToHost);
    cudaMemcpy(b.data(), B.d[2], sizeof(double) * kN, cudaMemcpyDeviceToHost);
    double ey = 0, ei = 0;
    for (int i = 0; i < kN; ++i) {
      const double m2 = mag2(ld3(&in[3 * i]));
      ey = std::fmax(ey, (double)std::fabs(a[i] * std::sqrt((long double)m2) - 1.0L));
      ei = std::fmax(ei, (double)std::fabs(b[i] * (long double)m2 - 1.0L));
    }
    std::printf("roots %d: wrong bits %llu, 1/sqrt %.3g, 1/a %.3g\n", kind, bad, ey, ei);
    fail += bad != 0 || !(ey <= 1.7e-16) || !(ei <= 1.2e-16);
  }
  // phases evenly over their logarithm, both signs, and near multiples of pi/2
  for (int kind = 0; kind < 3; ++kind) {
    for (int i = 0; i < kN; ++i) {
      const double e = kind == 0 ? std::exp2(23.0 + 23.0 * U(rng)) : std::exp2(48.0 + 2.0 * U(rng));
      in[i] = kind < 2 ? std::copysign(e, U(rng))
                       : (double)std::rint((long double)std::exp2(22.0 + 22.0 * U(rng))) * 1.5707963267948966 +
                             1e-7 * U(rng);
    }
    cudaMemcpy(B.d[0], in.data(), sizeof(double) * kN, cudaMemcpyHostToDevice);
    sines<<<kN / 128, 128>>>(B.d[0], kN, B.d[1], B.d[2]);
    cudaMemcpy(a.data(), B.d[1], sizeof(double) * kN, cudaMemcpyDeviceToHost);
    cudaMemcpy(b.data(), B.d[2], sizeof(double) * kN, cudaMemcpyDeviceToHost);
    double es = 0, ec = 0;
    for (int i = 0; i < kN; ++i) {
      es = std::fmax(es, (double)std::fabs(a[i] - std::sin((long double)in[i])));
      ec = std::fmax(ec, (double)std::fabs(b[i] - std::cos((long double)in[i])));
    }
    const double tol = kind == 1 ? 4e-16 : 2.4e-16;
    std::printf("sines %d: sin %.3g, cos %.3g of %.3g\n", kind, es, ec, tol);
    fail += !(es <= tol) || !(ec <= tol);
  }
  const cudaError_t e = cudaDeviceSynchronize();
  std::printf("%s, bad %d\n", cudaGetErrorString(e), fail);
  return fail != 0 || e != cudaSuccess;
}
