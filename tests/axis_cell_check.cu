// Host-side check of axis_cell, the cell of a one-axis field map (run by tests/test_axis_cell_cpu.py): for every
// quotient the same cell as the general interpolation's conversion to an unsigned 64-bit number and limit, with
// that conversion's results for negative numbers and NaN (0 and 2^63) written out, and never outside the map.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <random>

#include "rk4_fields.cuh"

static int general(double q, int last) {
  const uint64_t k = q != q ? 1ull << 63 : q <= 0 ? 0 : q >= 0x1p64 ? ~0ull : (uint64_t)q;
  return k > (uint64_t)last ? last : (int)k;
}

int main() {
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  std::mt19937_64 rng(3);
  int bad = 0;
  for (int last : {0, 1, 2, 699, 1999, (1 << 30) - 3}) {
    auto check = [&](double q) {
      const int k = srs::axis_cell(q, last);
      if (k < 0 || k > last || k != general(q, last)) {
        std::printf("quotient %g of %d: cell %d\n", q, last, k);
        ++bad;
      }
    };
    for (double q : {nan, -nan, inf, -inf, 0.0, -0.0, 5e-324, -5e-324, -1.0, -1e300, 1e300, 0x1p31, 0x1p32, 0x1p63, 0x1p64})
      check(q);
    for (int d = -2; d <= 2; ++d) {
      check((double)last + d);
      check(std::nextafter((double)last + d, inf));
      check(std::nextafter((double)last + d, -inf));
    }
    std::uniform_real_distribution<double> U(-1.0, last + 2.0);
    for (int k = 0; k < 100000; ++k) check(U(rng));
  }
  std::printf("bad %d\n", bad);
  return bad != 0;
}
