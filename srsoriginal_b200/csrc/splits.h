// What the launchers that split a sum over CTAs ask of the device.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>

namespace srs {

// Resident CTAs of `kernel` (`threads` threads, no dynamic shared memory) on the current device, queried
// once per (kernel, device, threads): the launchers ask on every call.
template <typename K>
inline int64_t wave_slots(K kernel, int threads) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, int, int>, int64_t> cache;
  int dev = 0, sms = 148, occ = 1;
  const bool have_dev = cudaGetDevice(&dev) == cudaSuccess;
  const auto key = std::make_tuple(reinterpret_cast<const void *>(kernel), dev, threads);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
  }
  if (have_dev) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, 0) != cudaSuccess || occ < 1) occ = 1;
  const int64_t slots = (int64_t)sms * occ;
  if (have_dev) {
    std::lock_guard<std::mutex> lk(mu);
    cache[key] = slots;
  }
  return slots;
}

}  // namespace srs
