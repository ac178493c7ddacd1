// rgf_fft_cache.h -- what a context's cached scratch and cuFFT plans belong to
// (host only, no CUDA).  A call runs on the caller's current device, which may
// differ from call to call, and either form may have used the cache last, so
// the scratch and the plans each carry their own device.
#pragma once
#include <cstddef>
#include <cstdint>

namespace rgf {

struct FftPlanKey {
  int dev = -1;
  int64_t nky = 0, nkz = 0, N = 0, chunk = 0, tail = 0;
  bool operator==(const FftPlanKey& o) const {
    return dev == o.dev && nky == o.nky && nkz == o.nkz && N == o.N && chunk == o.chunk && tail == o.tail;
  }
};

struct FftKeys {
  int scratch_dev = -1;
  std::size_t scratch_bytes = 0;
  FftPlanKey plans;
  bool scratch_fits(int dev, std::size_t need) const { return scratch_dev == dev && scratch_bytes >= need; }
  bool plans_fit(const FftPlanKey& k) const { return plans.dev >= 0 && plans == k; }
  void set_scratch(int dev, std::size_t bytes) {
    scratch_dev = dev;
    scratch_bytes = bytes;
  }
  void set_plans(const FftPlanKey& k) { plans = k; }
  void drop_plans() { plans = FftPlanKey(); }
};

}  // namespace rgf
