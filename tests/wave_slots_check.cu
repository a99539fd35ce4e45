// wave_slots on a GPU (run by tests/test_gpu_units.py): the resident blocks of one kernel for several block sizes, asked
// twice each, are the occupancy calculator's.
#include <cstdio>

#include "splits.h"

__global__ void kernel(int *p) { *p = threadIdx.x; }

int main() {
  int dev = 0, sms = 0, bad = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int twice = 0; twice < 2; ++twice)
    for (int threads : {64, 128, 1024, 256}) {
      int occ = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, 0);
      const long long got = srs::wave_slots(kernel, threads);
      if (occ < 1 || got != (long long)sms * occ) {
        std::printf("%d threads: %lld, not %d x %d\n", threads, got, sms, occ);
        ++bad;
      }
    }
  std::printf("bad %d\n", bad);
  return bad != 0;
}
