// Exact sample medians on the device by radix select over monotone uint32 keys
// (float_key): the element of rank count / 2, the value std::nth_element(count
// / 2) returns. Shared by the subtraction's fill values (src/subtract.cpp:20-51,
// 915-945) and stamp selection's background and MAD (src/detect.cpp:100-112).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace dgpu {

// One sample: the finite values v[j * step] whose mask byte is 0 (any value when
// mask is null).
struct MedianJob {
  const float* v = nullptr;
  const uint8_t* mask = nullptr;
  int64_t n = 0, step = 1;
  float* out = nullptr;       // [0] the upper median (0 for an empty sample)
  int mad = 0;                // 1: out[1] = the upper median of |value - out[0]|
  unsigned* clear = nullptr;  // counters to zero on the way (see nclear)
  int nclear = 0;
};

// Samples of one launch: up to two (the two images of a pair).
constexpr int kMedianJobs = 2;
// Largest sample launch_medians takes.
constexpr int64_t kMedianMax = int64_t(1) << 19;

// scratch: medians_scratch bytes of device memory.
size_t medians_scratch(const MedianJob* jobs, int njobs);
void launch_medians(cudaStream_t s, const MedianJob* jobs, int njobs, void* scratch);

// *out = the upper median of a sample of any size.
void launch_upper_median(Context& c, int64_t n, int64_t step, const float* v, const uint8_t* mask, float* out);

}  // namespace dgpu
