// Stamp selection on the device (reference src/detect.cpp:84-314) and the
// median PSF stamp of the score path (python/delta/pipeline.py:285-302).
//
//  * background: median and 1.4826 * MAD of a flat-index-strided sample of the
//    finite, unmasked pixels (step n / 2^18), by exact radix select;
//  * peaks: 3x3 strict local maxima above median + k sigma inside the border,
//    with a fully on-frame, finite, unmasked, unsaturated stamp footprint;
//  * per-candidate flux-weighted second-moment FWHM (FP64);
//  * candidates sorted by flux descending (raster index ascending on ties),
//    then brightest-first greedy isolation, both in one CTA.
// Both images of a pair go through each launch together, and nothing is read
// back until the kept stamps are measured.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <string>

#include "dev_common.cuh"
#include "select_internal.h"
#include "detect_internal.h"

namespace dgpu {

// The background sample of an image: about 2^18 pixels at a fixed flat step;
// out[0] = median, out[1] = MAD (src/detect.cpp:100-112).
static MedianJob background_job(int64_t n, const float* img, const uint8_t* mask, float* out) {
  constexpr int64_t kTarget = 1 << 18;
  MedianJob j;
  j.v = img;
  j.mask = mask;
  j.n = n;
  j.step = n > kTarget ? n / kTarget : 1;
  j.out = out;
  j.mad = 1;
  return j;
}

// ---------------------------------------------------------------------------
// Candidates
// ---------------------------------------------------------------------------
__device__ bool footprint_ok_dev(const float* img, const uint8_t* mask, int w, int h, int x, int y, int r,
                                 double sat) {
  if (x - r < 0 || x + r >= w || y - r < 0 || y + r >= h) return false;
  for (int dy = -r; dy <= r; ++dy)
    for (int dx = -r; dx <= r; ++dx) {
      const size_t i = static_cast<size_t>(y + dy) * w + (x + dx);
      const float v = img[i];
      if (!isfinite(v)) return false;
      if (mask && mask[i] != 0) return false;
      if (sat > 0.0 && static_cast<double>(v) >= sat) return false;
    }
  return true;
}

// estimate_fwhm (src/detect.cpp:115-157), FP64.
__device__ double fwhm_dev(const float* img, int w, int h, int x, int y, int r, double bg) {
  double sum = 0.0, sx = 0.0, sy = 0.0;
  for (int dy = -r; dy <= r; ++dy) {
    const int yy = y + dy;
    if (yy < 0 || yy >= h) continue;
    for (int dx = -r; dx <= r; ++dx) {
      const int xx = x + dx;
      if (xx < 0 || xx >= w) continue;
      const double f = static_cast<double>(img[static_cast<size_t>(yy) * w + xx]) - bg;
      const double wt = f > 0.0 ? f : 0.0;
      sum += wt;
      sx += wt * dx;
      sy += wt * dy;
    }
  }
  if (sum <= 0.0) return __longlong_as_double(0x7ff8000000000000ll);
  const double mx = sx / sum, my = sy / sum;
  double sxx = 0.0, syy = 0.0;
  for (int dy = -r; dy <= r; ++dy) {
    const int yy = y + dy;
    if (yy < 0 || yy >= h) continue;
    for (int dx = -r; dx <= r; ++dx) {
      const int xx = x + dx;
      if (xx < 0 || xx >= w) continue;
      const double f = static_cast<double>(img[static_cast<size_t>(yy) * w + xx]) - bg;
      const double wt = f > 0.0 ? f : 0.0;
      sxx += wt * (dx - mx) * (dx - mx);
      syy += wt * (dy - my) * (dy - my);
    }
  }
  const double var = 0.5 * (sxx / sum + syy / sum);
  if (var <= 0.0) return __longlong_as_double(0x7ff8000000000000ll);
  return 2.354820045030949 * sqrt(var);
}

// One image of a launch over up to two.
struct DetectDev {
  const float* img;
  const uint8_t* mask;
  const float* bg;    // median, MAD
  unsigned* count;    // [0] candidates, [1] 3x3 peaks, [2] kept, [3] 1: too many candidates for the fast path
  int* peaks;         // raster indices
  int* cand;          // peaks whose stamp footprint is usable
  int* kept;          // max_stamps
  double* props;      // 3 x max_stamps: flux, S/N, FWHM
};
struct DetectPair {
  DetectDev d[kMedianJobs];
};

// 3x3 maxima above the threshold, 256 adjacent pixels of a row per warp. The
// comparisons are those of the FP64 values: v > t for a float v and a double t
// is v > (the largest float <= t). Bound by reading the image (4 bytes a pixel).
constexpr int kPeakSpan = 256;

__global__ void __launch_bounds__(256) k_peaks(int w, int h, DetectPair jobs, DetectParamsDev p, int cap) {
  const DetectDev j = jobs.d[blockIdx.y];
  const double med = static_cast<double>(j.bg[0]);
  const double sigma = 1.4826 * static_cast<double>(j.bg[1]);
  const double thr = med + p.threshold_sigma * (sigma > 0.0 ? sigma : 1.0);
  float t = static_cast<float>(thr);
  if (static_cast<double>(t) > thr) t = nextafterf(t, -INFINITY);
  const int b = max(p.border, 1);  // and the 3x3 window on the frame
  const int lane = threadIdx.x & 31, spans = (w + kPeakSpan - 1) / kPeakSpan;
  const int warps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
  for (int64_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < static_cast<int64_t>(spans) * h; s += warps) {
    const int y = static_cast<int>(s / spans), x0 = static_cast<int>(s - static_cast<int64_t>(y) * spans) * kPeakSpan + lane;
    if (y < b || y >= h - b) continue;
    const float* row = j.img + static_cast<size_t>(y) * w;
    float v[kPeakSpan / 32];
#pragma unroll
    for (int u = 0; u < kPeakSpan / 32; ++u) v[u] = x0 + 32 * u < w ? __ldg(row + x0 + 32 * u) : 0.0f;
#pragma unroll
    for (int u = 0; u < kPeakSpan / 32; ++u) {
      const int x = x0 + 32 * u;
      if (x < b || x >= w - b || !(v[u] > t)) continue;
      bool peak = true;
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
          if ((dx != 0 || dy != 0) && __ldg(row + static_cast<int64_t>(dy) * w + x + dx) > v[u]) peak = false;
      if (!peak) continue;
      const unsigned slot = atomicAdd(j.count + 1, 1u);
      if (static_cast<int>(slot) < cap) j.peaks[slot] = y * w + x;
    }
  }
}

// Stamp footprint of every 3x3 peak, one warp per peak: fully on the frame,
// finite, unmasked and below saturation (src/detect.cpp:190-214). Eight rows are
// in flight at a time.
__global__ void __launch_bounds__(256) k_footprint(int w, int h, DetectPair jobs, DetectParamsDev p, int cap) {
  const DetectDev j = jobs.d[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const int nwarp = static_cast<int>((gridDim.x * blockDim.x) >> 5);
  const int np = min(static_cast<int>(j.count[1]), cap);
  const int r = p.stamp_radius;
  for (int c = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < np; c += nwarp) {
    const int i = j.peaks[c];
    const int x = i % w, y = i / w;
    if (x - r < 0 || x + r >= w || y - r < 0 || y + r >= h) continue;
    bool ok = true;
    for (int dy = -r; dy <= r && ok; dy += 8) {
      for (int dx = lane - r; dx <= r; dx += 32) {
        float v[8];
        uint8_t m[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const size_t at = static_cast<size_t>(y + min(dy + u, r)) * w + (x + dx);
          v[u] = __ldg(j.img + at);
          m[u] = j.mask ? __ldg(j.mask + at) : 0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (!isfinite(v[u]) || m[u] != 0 || (p.saturation > 0.0 && static_cast<double>(v[u]) >= p.saturation)) ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok && lane == 0) {
      const unsigned slot = atomicAdd(j.count, 1u);
      if (static_cast<int>(slot) < cap) j.cand[slot] = i;
    }
  }
}

// (flux descending, index ascending) as an ascending uint64.
__device__ __forceinline__ unsigned long long cand_key(float v, int idx) {
  return (static_cast<unsigned long long>(~float_key(v)) << 32) | static_cast<unsigned>(idx);
}

__global__ void k_cand_keys(const unsigned* count, int cap, const int* __restrict__ cand, const float* __restrict__ img,
                            unsigned long long* __restrict__ keys, int* __restrict__ vals) {
  const int nc = min(static_cast<int>(*count), cap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nc; i += gridDim.x * blockDim.x) {
    const int idx = cand[i];
    keys[i] = cand_key(img[idx], idx);
    vals[i] = idx;
  }
}

// Brightest-first greedy isolation (src/detect.cpp:223-240) by one CTA of 1024
// threads, chunk by chunk of at most 1024 candidates in order, a thread to each.
// The kept stamps, and the chunk's candidates that none of those excludes, hang
// on lists hashed by cells of the isolation radius, so that a candidate looks at
// nine cells only. In each round a candidate looks for a brighter neighbour that
// is kept (it is out) or undecided (it waits there, and goes on from there when
// that one is out); if none is left it is kept. The rounds follow the longest
// chain of waiting candidates, 3 to 5 on star fields; the brightest undecided
// candidate always decides, so 1024 bound them. Where a frame has room for few
// stamps (few_stamps) the chunk keeps one a round instead.
constexpr int kIsoHeads = 1024;
struct Isolation {
  int4 node[1024];  // x, y, next
  int head[kIsoHeads], khead[kIsoHeads];
  unsigned char state[1024];
  int wsum[32];
  int4 first[2][32];  // each warp's brightest undecided candidate: thread, x, y
};
__device__ __forceinline__ int iso_bucket(int cx, int cy) {
  return static_cast<int>((static_cast<unsigned>(cx) * 0x9E3779B1u ^ static_cast<unsigned>(cy) * 0x85EBCA6Bu) >> 22);
}
// Dynamic shared memory of the kept stamps: x, y and the next of each.
__host__ __device__ constexpr size_t iso_smem(int max_stamps) {
  return (2 * sizeof(int) + sizeof(uint16_t)) * static_cast<size_t>(max_stamps > 1 ? max_stamps : 1);
}
__device__ __forceinline__ bool iso_near(int dx, int dy, int r, long long r2) {
  dx = abs(dx);
  dy = abs(dy);
  if (dx >= r || dy >= r) return false;
  const long long lx = dx, ly = dy;
  return lx * lx + ly * ly < r2;
}

// One chunk: thread t < n holds raster index idx. Returns the number kept so far.
__device__ int isolate_chunk(Isolation& sh, int w, int n, int idx, int iso, bool few, int max_stamps, int nk, int* ks,
                             int* __restrict__ kept) {
  enum : unsigned char { kOut, kKept, kOpen };
  volatile unsigned char* state = sh.state;
  uint16_t* knext = reinterpret_cast<uint16_t*>(ks + 2 * (max_stamps > 1 ? max_stamps : 1));
  constexpr int kEnd = 0xffff;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = abs(iso), cell = max(1, r);
  const long long r2 = static_cast<long long>(r) * r;
  const int x = idx % w, y = idx / w, cx = x / cell, cy = y / cell;
  for (int i = tid; i < kIsoHeads; i += 1024) {
    sh.head[i] = kEnd;
    if (nk == 0) sh.khead[i] = kEnd;
  }
  __syncthreads();
  bool open = tid < n;
  if (nk > 0)
    for (int q = 0; q < 9 && open; ++q)
      for (int k = sh.khead[iso_bucket(cx - 1 + q % 3, cy - 1 + q / 3)]; k != kEnd && open; k = knext[k])
        open = !iso_near(x - ks[2 * k], y - ks[2 * k + 1], r, r2);
  bool mine = false;
  if (few) {
    // Round by round the brightest candidate left is kept and the others drop out that
    // lie near it.
    for (int round = 0, left = max_stamps - nk; round < left; ++round) {
      const unsigned vote = __ballot_sync(0xffffffffu, open);
      if (vote ? lane == __ffs(vote) - 1 : lane == 0) sh.first[round & 1][warp] = make_int4(vote ? tid : 1024, x, y, 0);
      __syncthreads();
      const int4 f = sh.first[round & 1][lane];
      const int best = __reduce_min_sync(0xffffffffu, f.x);
      if (best == 1024) break;
      const int from = best >> 5;
      const int bx = __shfl_sync(0xffffffffu, f.y, from), by = __shfl_sync(0xffffffffu, f.z, from);
      if (best == tid) mine = true;
      open = open && best != tid && !iso_near(x - bx, y - by, r, r2);
    }
    open = false;
  }
  state[tid] = open ? kOpen : kOut;
  if (open) sh.node[tid] = make_int4(x, y, atomicExch(&sh.head[iso_bucket(cx, cy)], tid), 0);
  __syncthreads();
  int q = 0, k = open ? sh.head[iso_bucket(cx - 1, cy - 1)] : kEnd;
  do {
    while (open) {
      if (k == kEnd) {
        if (++q == 9) {
          mine = true;
          open = false;
          state[tid] = kKept;
          break;
        }
        const int row = q >= 6 ? 2 : q >= 3 ? 1 : 0;
        k = sh.head[iso_bucket(cx - 1 + q - 3 * row, cy - 1 + row)];
        continue;
      }
      const int4 c = sh.node[k];
      if (k < tid && iso_near(x - c.x, y - c.y, r, r2)) {
        const unsigned char st = state[k];
        if (st == kOpen) break;
        if (st == kKept) {
          open = false;
          state[tid] = kOut;
          break;
        }
      }
      k = c.z;
    }
  } while (__syncthreads_or(open));
  const unsigned vote = __ballot_sync(0xffffffffu, mine);
  if (lane == 0) sh.wsum[warp] = __popc(vote);
  __syncthreads();
  const int c = sh.wsum[lane];
  int at = nk + __popc(vote & ((1u << lane) - 1u)) + __reduce_add_sync(0xffffffffu, lane < warp ? c : 0);
  if (mine && at < max_stamps) {
    ks[2 * at] = x;
    ks[2 * at + 1] = y;
    kept[at] = idx;
    knext[at] = static_cast<uint16_t>(atomicExch(&sh.khead[iso_bucket(cx, cy)], at));
  }
  nk = min(nk + __reduce_add_sync(0xffffffffu, c), max_stamps);
  __syncthreads();
  return nk;
}

// Ascending bitonic sort of 1024 keys, one per thread: exchanges within a warp by
// shuffles, only the longer ones through shared memory. Returns the thread's key.
__device__ unsigned long long sort_1024(unsigned long long k, unsigned long long* sk) {
  const int tid = threadIdx.x;
  for (int size = 2; size <= 1024; size <<= 1)
    for (int half = size >> 1; half > 0; half >>= 1) {
      unsigned long long other;
      if (half >= 32) {
        __syncthreads();
        sk[tid] = k;
        __syncthreads();
        other = sk[tid ^ half];
      } else {
        other = __shfl_xor_sync(0xffffffffu, k, half);
      }
      const bool least = ((tid & size) == 0) == ((tid & half) == 0);
      if (least == (other < k)) k = other;
    }
  return k;
}

// Sort and isolation of one image's candidates in one CTA, which holds up to
// kSortMost keys. Only the chunks that isolation asks for are sorted: each time
// the brightest keys left, 512 to 1024 of them, are found on a histogram of the
// range that is left (and of the bin where it passes 1024, if there are fewer
// than 512 below that), gathered and sorted. With max_stamps of a few hundred one
// or two chunks do, however many candidates there are. More candidates set
// count[3] (the host then takes the general path). Keys to global memory, a radix
// sort and an isolation by single warps took 4 to 20 launches and 110 to 190 us
// per image (2000 to 8400 candidates); this launch takes 40 us for both images
// (770 and 1650 candidates at 1003x1531, 8400 at 4096x4096; 52 and 212 us when it
// sorted all keys).
constexpr int kSortMost = 16384;
constexpr int kSortStamps = 4096;  // the most stamps whose places fit beside the keys
constexpr int kIsoStamps = 20480;  // and the most that fit without the keys

__global__ void __launch_bounds__(1024) k_sort_isolate(int w, DetectPair jobs, int iso, bool few, int max_stamps) {
  using u64 = unsigned long long;
  extern __shared__ __align__(16) u64 keys[];
  __shared__ Isolation sh;
  __shared__ u64 chunk[1024];
  __shared__ int hist[1024];
  __shared__ u64 s_lo, s_hi;
  __shared__ int s_sum[32], s_n, s_bin, s_below;
  const DetectDev j = jobs.d[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nc = static_cast<int>(min(j.count[0], static_cast<unsigned>(kSortMost) + 1u));
  if (nc > kSortMost) {
    if (tid == 0) j.count[3] = 1u;
    return;
  }
  if (tid == 0) {
    s_lo = ~0ull;
    s_hi = 0;
  }
  __syncthreads();
  u64 lo = ~0ull, hi = 0;
  for (int i = tid; i < nc; i += 1024) {
    const int idx = j.cand[i];
    const u64 k = cand_key(__ldg(j.img + idx), idx);
    keys[i] = k;
    lo = min(lo, k);
    hi = max(hi, k);
  }
  for (int d = 16; d > 0; d >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
  }
  if (lane == 0) {
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
  }
  __syncthreads();
  lo = s_lo;
  const u64 last = s_hi;  // keys in [lo, last] are left
  int* ks = reinterpret_cast<int*>(keys + kSortMost);
  int nk = 0;
  for (int left = nc; left > 0 && nk < max_stamps;) {
    // end: one past the chunk's greatest key. [lo, from) is in the chunk, n keys.
    u64 end = last, from = lo, to = last;
    int n = 0;
    if (left > 1024) {
      while (true) {
        const int shift = max(0, 64 - __clzll(static_cast<long long>(to - from)) - 10);  // (to - from) >> shift < 1024
        hist[tid] = 0;
        __syncthreads();
        for (int i = tid; i < nc; i += 1024) {
          const u64 k = keys[i];
          if (k >= from && k <= to) atomicAdd(&hist[(k - from) >> shift], 1);
        }
        __syncthreads();
        int sum = hist[tid];
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, sum, d);
          if (lane >= d) sum += o;
        }
        if (lane == 31) s_sum[warp] = sum;
        __syncthreads();
        sum += __reduce_add_sync(0xffffffffu, lane < warp ? s_sum[lane] : 0);
        const int before = sum - hist[tid];
        if (n + before <= 1024 && n + sum > 1024) {  // one bin: more than 1024 keys are left
          s_bin = tid;
          s_below = before;
        }
        __syncthreads();
        n += s_below;
        from += static_cast<u64>(s_bin) << shift;
        to = min(to, from + (((1ull << shift) - 1)));
        end = from - 1;
        if (n >= 512) break;
      }
    } else {
      n = left;
    }
    if (tid == 0) s_n = 0;
    __syncthreads();
    for (int i = tid; i < nc; i += 1024) {
      const u64 k = keys[i];
      if (k >= lo && k <= end) chunk[atomicAdd(&s_n, 1)] = k;
    }
    __syncthreads();
    const u64 k = sort_1024(tid < n ? chunk[tid] : ~0ull, chunk);
    nk = isolate_chunk(sh, w, n, tid < n ? static_cast<int>(k & 0xffffffffull) : 0, iso, few, max_stamps, nk, ks, j.kept);
    lo = end + 1;
    left -= n;
  }
  if (tid == 0) j.count[2] = static_cast<unsigned>(nk);
}

// Isolation of candidates sorted in global memory.
__global__ void __launch_bounds__(1024)
k_isolate(int w, DetectDev j, int cap, const int* __restrict__ sorted_idx, int iso, bool few, int max_stamps) {
  extern __shared__ int ks[];
  __shared__ Isolation sh;
  const int nc = min(static_cast<int>(j.count[0]), cap);
  int nk = 0;
  for (int base = 0; base < nc && nk < max_stamps; base += 1024) {
    const int n = min(nc - base, 1024);
    const int idx = static_cast<int>(threadIdx.x) < n ? sorted_idx[base + threadIdx.x] : 0;
    nk = isolate_chunk(sh, w, n, idx, iso, few, max_stamps, nk, ks, j.kept);
  }
  if (threadIdx.x == 0) j.count[2] = static_cast<unsigned>(nk);
}

// One CTA per kept stamp: the threads stage the clipped weights
// max(f - bg, 0) of the FWHM window in shared memory (0 off the frame, which
// adds an exact zero where the reference skips the pixel), then thread 0 runs
// the two FP64 moment passes of fwhm_dev in the same (dy, dx) order.
__global__ void __launch_bounds__(256) k_stamp_props(int w, int h, DetectPair jobs, int fwhm_radius, int max_stamps) {
  extern __shared__ double wt[];  // (2r+1)^2
  const DetectDev j = jobs.d[blockIdx.y];
  const int i = blockIdx.x;
  if (i >= static_cast<int>(j.count[2])) return;
  const float* img = j.img;
  double *flux = j.props, *snr = flux + max_stamps, *fwhm = snr + max_stamps;
  const double med = static_cast<double>(j.bg[0]);
  const double sigma = 1.4826 * static_cast<double>(j.bg[1]);
  const int idx = j.kept[i];
  const int x = idx % w, y = idx / w;
  const int r = fwhm_radius, side = 2 * r + 1;
  for (int e = threadIdx.x; e < side * side; e += blockDim.x) {
    const int yy = y - r + e / side, xx = x - r + e % side;
    double v = 0.0;
    if (yy >= 0 && yy < h && xx >= 0 && xx < w) {
      const double f = static_cast<double>(img[static_cast<size_t>(yy) * w + xx]) - med;
      v = f > 0.0 ? f : 0.0;
    }
    wt[e] = v;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const double f0 = static_cast<double>(img[idx]) - med;
  flux[i] = f0;
  snr[i] = sigma > 0.0 ? f0 / sigma : f0;
  double sum = 0.0, sx = 0.0, sy = 0.0;
  for (int dy = -r; dy <= r; ++dy)
    for (int dx = -r; dx <= r; ++dx) {
      const double wv = wt[(dy + r) * side + dx + r];
      sum += wv;
      sx += wv * dx;
      sy += wv * dy;
    }
  double out = __longlong_as_double(0x7ff8000000000000ll);
  if (sum > 0.0) {
    const double mx = sx / sum, my = sy / sum;
    double sxx = 0.0, syy = 0.0;
    for (int dy = -r; dy <= r; ++dy)
      for (int dx = -r; dx <= r; ++dx) {
        const double wv = wt[(dy + r) * side + dx + r];
        sxx += wv * (dx - mx) * (dx - mx);
        syy += wv * (dy - my) * (dy - my);
      }
    const double var = 0.5 * (sxx / sum + syy / sum);
    if (var > 0.0) out = 2.354820045030949 * sqrt(var);
  }
  fwhm[i] = out;
}

// Catalog positions: footprint check on both images + FWHM on both
// (select_stamps_from_catalog, src/detect.cpp:289-314).
__global__ void k_catalog_stamps(int w, int h, const float* __restrict__ sci, const uint8_t* __restrict__ sm,
                                 const float* __restrict__ ref, const uint8_t* __restrict__ rm,
                                 const float* __restrict__ bg_sci, const float* __restrict__ bg_ref,
                                 const int* __restrict__ xs, const int* __restrict__ ys, int n, DetectParamsDev p,
                                 int* __restrict__ ok, double* __restrict__ fs, double* __restrict__ fr) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int x = xs[i], y = ys[i];
    const bool good = footprint_ok_dev(sci, sm, w, h, x, y, p.stamp_radius, p.saturation) &&
                      footprint_ok_dev(ref, rm, w, h, x, y, p.stamp_radius, p.saturation);
    ok[i] = good ? 1 : 0;
    if (good) {
      fs[i] = fwhm_dev(sci, w, h, x, y, p.fwhm_radius, static_cast<double>(bg_sci[0]));
      fr[i] = fwhm_dev(ref, w, h, x, y, p.fwhm_radius, static_cast<double>(bg_ref[0]));
    }
  }
}

// Median unit-sum PSF of the listed stamps (python/delta/pipeline.py:285-302):
// per stamp cut - median(cut) normalised by its positive total; per pixel the
// median across stamps (mean of the two middle values for an even count),
// clipped at 0 and renormalised. FP64. One CTA per stamp, then one per pixel.
__global__ void k_psf_stamps(int w, int h, const float* __restrict__ img, const int* __restrict__ xs,
                             const int* __restrict__ ys, int n, int radius, double* __restrict__ cuts,
                             int* __restrict__ use) {
  extern __shared__ double sv[];  // side^2 padded to a power of two
  const int s = blockIdx.x;
  const int side = 2 * radius + 1, np = side * side;
  int cap = 1;
  while (cap < np) cap <<= 1;
  const int x = xs[s], y = ys[s];
  const bool inside = !(x - radius < 0 || x + radius >= w || y - radius < 0 || y + radius >= h);
  if (!inside) {
    if (threadIdx.x == 0) use[s] = 0;
    return;
  }
  double* srt = sv + cap;
  for (int i = threadIdx.x; i < cap; i += blockDim.x) {
    double v = INFINITY;
    if (i < np) v = static_cast<double>(img[static_cast<size_t>(y - radius + i / side) * w + (x - radius + i % side)]);
    sv[i] = v;
    srt[i] = v;
  }
  __syncthreads();
  for (int size = 2; size <= cap; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < cap; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const double a = srt[i], b = srt[j];
          if ((a > b) == up) {
            srt[i] = b;
            srt[j] = a;
          }
        }
      }
      __syncthreads();
    }
  const double med = (np & 1) ? srt[np / 2] : 0.5 * (srt[np / 2 - 1] + srt[np / 2]);
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int i = 0; i < np; ++i) tot += sv[i] - med;
    use[s] = tot > 0.0 ? 1 : 0;
    srt[0] = tot;
  }
  __syncthreads();
  const double tot = srt[0];
  for (int i = threadIdx.x; i < np; i += blockDim.x) cuts[static_cast<size_t>(s) * np + i] = (sv[i] - med) / tot;
}

// Median over the used stamps of pixel p (a CTA per pixel): each used value's
// rank among the used values (ties broken by stamp index) is counted in
// parallel; the values of rank cnt/2 (and cnt/2 - 1) give the median.
__global__ void __launch_bounds__(256) k_psf_median(int n, int np, const double* __restrict__ cuts,
                                                     const int* __restrict__ use, double* __restrict__ out,
                                                     unsigned* status) {
  extern __shared__ double col[];
  int* used = reinterpret_cast<int*>(col + n);
  const int p = blockIdx.x;
  __shared__ int cnt;
  __shared__ double lo, hi;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  int mine = 0;
  for (int s = threadIdx.x; s < n; s += blockDim.x) {
    const int u = use[s] != 0;
    used[s] = u;
    col[s] = u ? cuts[static_cast<size_t>(s) * np + p] : 0.0;
    mine += u;
  }
  atomicAdd(&cnt, mine);
  __syncthreads();
  const int c = cnt;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    if (!used[i]) continue;
    const double v = col[i];
    int rank = 0;
    for (int j = 0; j < n; ++j)
      if (used[j] && (col[j] < v || (col[j] == v && j < i))) ++rank;
    if (rank == c / 2) hi = v;
    if (rank == c / 2 - 1) lo = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    if (c > 0) m = (c & 1) ? hi : 0.5 * (lo + hi);
    out[p] = m > 0.0 ? m : 0.0;
    if (c == 0) atomicOr(status, kStatusBounds);
  }
}

void launch_psf_estimate(Context& c, int w, int h, const float* img, const int* xs, const int* ys, int n, int radius,
                         double* out, int* n_used) {
  cudaStream_t s = c.stream;
  const int side = 2 * radius + 1, np = side * side;
  int cap = 1;
  while (cap < np) cap <<= 1;
  double* cuts = static_cast<double*>(c.slot(kSlotScratch0, sizeof(double) * static_cast<size_t>(std::max(n, 1)) * np));
  int* use = static_cast<int*>(c.slot(kSlotBlockCounts, sizeof(int) * std::max(n, 1)));
  const size_t smem = sizeof(double) * 2 * cap;
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_psf_stamps), smem);
  k_psf_stamps<<<n, 256, smem, s>>>(w, h, img, xs, ys, n, radius, cuts, use);
  DGPU_LAUNCH("k_psf_stamps");
  const size_t smem2 = (sizeof(double) + sizeof(int)) * std::max(n, 1);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_psf_median), smem2);
  k_psf_median<<<np, 256, smem2, s>>>(n, np, cuts, use, out, c.d_status);
  DGPU_LAUNCH("k_psf_median");
  std::vector<int> hu(n);
  if (n) read_back(c, hu.data(), use, sizeof(int) * n);
  sync_reads(c);
  int u = 0;
  for (int v : hu) u += v;
  *n_used = u;
}

// weighted_mean (src/bindings.cpp:107-124): FP64 partial sums per CTA.
__global__ void k_weighted_mean(int64_t n, const float* __restrict__ d, const float* __restrict__ v,
                                const uint8_t* __restrict__ m, double* __restrict__ part) {
  __shared__ double s1[256], s2[256];
  double a = 0.0, b = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (m[i] != 0) continue;
    if (!(v[i] > 0.0f)) continue;
    const double wv = 1.0 / static_cast<double>(v[i]);
    a += wv;
    b += wv * static_cast<double>(d[i]);
  }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = b;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < static_cast<unsigned>(o)) {
      s1[threadIdx.x] += s1[threadIdx.x + o];
      s2[threadIdx.x] += s2[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s1[0];
    part[2 * blockIdx.x + 1] = s2[0];
  }
}

void launch_weighted_mean(Context& c, int64_t n, const float* d, const float* v, const uint8_t* m, double* out2) {
  const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 296));
  double* part = static_cast<double*>(c.slot(kSlotScratch1, sizeof(double) * 2 * blocks));
  k_weighted_mean<<<blocks, 256, 0, c.stream>>>(n, d, v, m, part);
  DGPU_LAUNCH("k_weighted_mean");
  std::vector<double> hp(2 * blocks);
  read_back(c, hp.data(), part, sizeof(double) * 2 * blocks);
  sync_reads(c);
  double a = 0.0, b = 0.0;
  for (int i = 0; i < blocks; ++i) {
    a += hp[2 * i];
    b += hp[2 * i + 1];
  }
  out2[0] = a;
  out2[1] = b;
}

// The detect pipeline of up to two images of one size.
struct DetectJob {
  const float* img;
  const uint8_t* mask;
  DetectHost* res;
  unsigned hc[4] = {0, 0, 0, 0};
  float hbg[2] = {0.0f, 0.0f};
  std::vector<int> hk;
  std::vector<double> props;
};
constexpr int kDetectCap = 1 << 20;

static void launch_stamp_props(cudaStream_t s, int w, int h, const DetectParamsDev& p, const DetectPair& jobs, int njobs,
                               int nstamps, int stride) {
  const size_t psmem = sizeof(double) * static_cast<size_t>(2 * p.fwhm_radius + 1) * (2 * p.fwhm_radius + 1);
  if (psmem > 200 * 1024) fail(DGPU_ERR_INVALID, "detect_stamps: fwhm_radius too large");
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_stamp_props), psmem);
  k_stamp_props<<<dim3(nstamps, njobs), 256, psmem, s>>>(w, h, jobs, p.fwhm_radius, stride);
  DGPU_LAUNCH("k_stamp_props");
}

// Whether isolation keeps few stamps: at most one in a square of side radius / sqrt 2,
// so (w / side + 1) (h / side + 1) bound them. Up to 640 the chunk is resolved a kept
// stamp at a time (0.3 us each): the cells of the lists then hold many candidates that
// wait for one another. 2000 stars at 1003 x 1531, up to 1000 stamps, by lists and by
// rounds: radius 50 (1302) 83 and 114 us, 80 (525) 122 and 63, 200 (118) 739 and 29;
// 8000 at 2048 x 2048: 80 (1384) 162 and 214, 120 (632) 189 and 149; 300 x 400 with 200
// stars: 20 (650) 22 and 37, 30 (300) 33 and 27, 200 (12) 1129 and 11.
static bool few_stamps(int w, int h, const DetectParamsDev& p) {
  const double side = std::abs(static_cast<double>(p.isolation_radius)) / std::sqrt(2.0);
  return side >= 1.0 && (w / side + 1.0) * (h / side + 1.0) <= 640.0;
}

// The general path of one image, for more candidates than one CTA sorts or more
// stamps than it keeps in shared memory beside them: radix sort, isolation and
// measurement, reading the kept count back in between. On entry j.hc[0] > 0.
static void detect_general(Context& c, int w, int h, const DetectParamsDev& p, DetectJob& j, const DetectDev& d) {
  cudaStream_t s = c.stream;
  const int cap = kDetectCap, nc = static_cast<int>(j.hc[0]);
  char* buf = static_cast<char*>(c.slot(kSlotFft2, (sizeof(int) * 2 + 2 * sizeof(unsigned long long)) * cap));
  auto* keys = reinterpret_cast<unsigned long long*>(buf);
  auto* keys2 = keys + cap;
  int* vals = reinterpret_cast<int*>(keys2 + cap);
  int* sorted = vals + cap;
  k_cand_keys<<<(nc + 255) / 256, 256, 0, s>>>(d.count, cap, d.cand, d.img, keys, vals);
  DGPU_LAUNCH("k_cand_keys");
  size_t tmp_bytes = 0;
  DGPU_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, vals, sorted, nc, 0, 64, s));
  void* tmp = c.slot(kSlotFft4, tmp_bytes + 16);
  DGPU_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, vals, sorted, nc, 0, 64, s));
  const size_t smem = iso_smem(p.max_stamps);
  if (p.max_stamps > kIsoStamps) fail(DGPU_ERR_INVALID, "detect_stamps: max_stamps above 20480 is not supported");
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_isolate), smem);
  k_isolate<<<1, 1024, smem, s>>>(w, d, cap, sorted, p.isolation_radius, few_stamps(w, h, p), p.max_stamps);
  DGPU_LAUNCH("k_isolate");
  read_back(c, j.hc, d.count, sizeof(j.hc));
  sync_reads(c);
  const int nk = static_cast<int>(j.hc[2]);
  if (nk <= 0) return;
  DetectPair one{};
  one.d[0] = d;
  one.d[0].props = static_cast<double*>(c.slot(kSlotCompOut, sizeof(double) * 3 * nk));
  launch_stamp_props(s, w, h, p, one, 1, nk, nk);
  j.hk.resize(nk);
  j.props.resize(3 * static_cast<size_t>(nk));
  read_back(c, j.hk.data(), d.kept, sizeof(int) * nk);
  read_back(c, j.props.data(), one.d[0].props, sizeof(double) * 3 * nk);
  sync_reads(c);
}

static void run_detect_jobs(Context& c, int w, int h, const DetectParamsDev& p, DetectJob* j, int njobs) {
  cudaStream_t s = c.stream;
  const int64_t n = static_cast<int64_t>(w) * h;
  const int cap = kDetectCap, most = std::max(p.max_stamps, 0);
  // In one CTA's shared memory: the sort keys and the kept stamps.
  const size_t sort_smem = sizeof(unsigned long long) * kSortMost + iso_smem(most);
  const size_t psmem = sizeof(double) * static_cast<size_t>(2 * p.fwhm_radius + 1) * (2 * p.fwhm_radius + 1);
  const bool fast = most <= kSortStamps && psmem <= 200 * 1024;
  // The general path keeps up to kIsoStamps (it refuses more) and measures elsewhere.
  const size_t kept_ints = (static_cast<size_t>(std::clamp(most, 1, kIsoStamps)) + 1) & ~size_t(1);
  const size_t per = 64 + sizeof(int) * (2 * static_cast<size_t>(cap) + kept_ints) +
                     sizeof(double) * 3 * (fast ? static_cast<size_t>(std::max(most, 1)) : 0);
  char* buf = static_cast<char*>(c.slot(kSlotFft0, per * njobs));
  DetectPair jobs{};
  MedianJob med[kMedianJobs];
  for (int i = 0; i < njobs; ++i) {
    DetectDev& d = jobs.d[i];
    char* b = buf + per * i;
    d.img = j[i].img;
    d.mask = j[i].mask;
    d.count = reinterpret_cast<unsigned*>(b);
    float* bg = reinterpret_cast<float*>(b + 32);
    d.bg = bg;
    d.peaks = reinterpret_cast<int*>(b + 64);
    d.cand = d.peaks + cap;
    d.kept = d.cand + cap;
    d.props = reinterpret_cast<double*>(d.kept + kept_ints);
    med[i] = background_job(n, d.img, d.mask, bg);
    med[i].clear = d.count;
    med[i].nclear = 4;
  }
  launch_medians(s, med, njobs, c.slot(kSlotSamples, medians_scratch(med, njobs)));
  const int64_t spans = static_cast<int64_t>((w + kPeakSpan - 1) / kPeakSpan) * h;
  k_peaks<<<dim3(static_cast<unsigned>(std::min<int64_t>((spans + 7) / 8, 148 * 8)), njobs), 256, 0, s>>>(w, h, jobs, p, cap);
  DGPU_LAUNCH("k_peaks");
  k_footprint<<<dim3(148 * 4, njobs), 256, 0, s>>>(w, h, jobs, p, cap);
  DGPU_LAUNCH("k_footprint");
  if (fast) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_sort_isolate), sort_smem);
    k_sort_isolate<<<njobs, 1024, sort_smem, s>>>(w, jobs, p.isolation_radius, few_stamps(w, h, p), p.max_stamps);
    DGPU_LAUNCH("k_sort_isolate");
    if (most > 0) launch_stamp_props(s, w, h, p, jobs, njobs, most, most);
  }
  for (int i = 0; i < njobs; ++i) {
    read_back(c, j[i].hc, jobs.d[i].count, sizeof(j[i].hc));
    read_back(c, j[i].hbg, jobs.d[i].bg, sizeof(j[i].hbg));
    if (fast && most > 0) {
      j[i].hk.resize(most);
      j[i].props.resize(3 * static_cast<size_t>(most));
      read_back(c, j[i].hk.data(), jobs.d[i].kept, sizeof(int) * most);
      read_back(c, j[i].props.data(), jobs.d[i].props, sizeof(double) * 3 * most);
    }
  }
  sync_reads(c);
  for (int i = 0; i < njobs; ++i) {
    if (j[i].hc[1] > static_cast<unsigned>(cap)) fail(DGPU_ERR_RUNTIME, "detect_stamps: more than 2^20 peak candidates");
    int stride = most;
    if (j[i].hc[0] > 0 && (!fast || j[i].hc[3] != 0)) {
      detect_general(c, w, h, p, j[i], jobs.d[i]);
      stride = static_cast<int>(j[i].hc[2]);
    }
    DetectHost& res = *j[i].res;
    res.median = static_cast<double>(j[i].hbg[0]);
    res.sigma = 1.4826 * static_cast<double>(j[i].hbg[1]);
    const int nk = static_cast<int>(j[i].hc[2]);
    res.x.resize(nk);
    res.y.resize(nk);
    res.flux.resize(nk);
    res.snr.resize(nk);
    res.fwhm.resize(nk);
    for (int q = 0; q < nk; ++q) {
      res.x[q] = j[i].hk[q] % w;
      res.y[q] = j[i].hk[q] / w;
      res.flux[q] = j[i].props[q];
      res.snr[q] = j[i].props[static_cast<size_t>(stride) + q];
      res.fwhm[q] = j[i].props[2 * static_cast<size_t>(stride) + q];
    }
  }
}

int run_detect(Context& c, int w, int h, const float* img, const uint8_t* mask, const DetectParamsDev& p,
               DetectHost& res) {
  DetectJob j;
  j.img = img;
  j.mask = mask;
  j.res = &res;
  run_detect_jobs(c, w, h, p, &j, 1);
  return static_cast<int>(res.x.size());
}

void run_detect_pair(Context& c, int w, int h, const float* img0, const uint8_t* mask0, const float* img1,
                     const uint8_t* mask1, const DetectParamsDev& p, DetectHost& res0, DetectHost& res1) {
  DetectJob j[2];
  j[0].img = img0;
  j[0].mask = mask0;
  j[0].res = &res0;
  j[1].img = img1;
  j[1].mask = mask1;
  j[1].res = &res1;
  run_detect_jobs(c, w, h, p, j, 2);
}

void run_background(Context& c, int64_t n, const float* img, const uint8_t* mask, double* median, double* sigma) {
  float* bg = static_cast<float*>(c.slot(kSlotFit14, 64));
  const MedianJob job = background_job(n, img, mask, bg);
  launch_medians(c.stream, &job, 1, c.slot(kSlotSamples, medians_scratch(&job, 1)));
  float hbg[2];
  read_back(c, hbg, bg, sizeof(hbg));
  sync_reads(c);
  *median = static_cast<double>(hbg[0]);
  *sigma = 1.4826 * static_cast<double>(hbg[1]);
}

void run_catalog_stamps(Context& c, int w, int h, const float* sci, const uint8_t* sm, const float* ref,
                        const uint8_t* rm, const int* xs_host, const int* ys_host, int n, const DetectParamsDev& p,
                        std::vector<int>& ok, std::vector<double>& fs, std::vector<double>& fr, double* med_sci,
                        double* med_ref) {
  cudaStream_t s = c.stream;
  const int64_t npx = static_cast<int64_t>(w) * h;
  float* bgs = static_cast<float*>(c.slot(kSlotFit14, 64));
  float* bgr = bgs + 2;
  const MedianJob jobs[2] = {background_job(npx, sci, sm, bgs), background_job(npx, ref, rm, bgr)};
  launch_medians(s, jobs, 2, c.slot(kSlotSamples, medians_scratch(jobs, 2)));
  int* dxy = static_cast<int*>(c.slot(kSlotBright, sizeof(int) * 2 * std::max(n, 1)));
  DGPU_CUDA(h2d_async(dxy, xs_host, sizeof(int) * n, s));
  DGPU_CUDA(h2d_async(dxy + n, ys_host, sizeof(int) * n, s));
  char* ob = static_cast<char*>(c.slot(kSlotCompStats, (sizeof(int) + 2 * sizeof(double)) * std::max(n, 1) + 64));
  double* dfs = reinterpret_cast<double*>(ob);
  double* dfr = dfs + std::max(n, 1);
  int* dok = reinterpret_cast<int*>(dfr + std::max(n, 1));
  if (n > 0) {
    k_catalog_stamps<<<(n + 127) / 128, 128, 0, s>>>(w, h, sci, sm, ref, rm, bgs, bgr, dxy, dxy + n, n, p, dok, dfs,
                                                     dfr);
    DGPU_LAUNCH("k_catalog_stamps");
  }
  ok.assign(n, 0);
  fs.assign(n, 0.0);
  fr.assign(n, 0.0);
  float hb[2];
  if (n) {
    read_back(c, ok.data(), dok, sizeof(int) * n);
    read_back(c, fs.data(), dfs, sizeof(double) * n);
    read_back(c, fr.data(), dfr, sizeof(double) * n);
  }
  read_back(c, hb, bgs, sizeof(float) * 2);
  sync_reads(c);
  *med_sci = hb[0];
  read_back(c, hb, bgr, sizeof(float) * 2);
  sync_reads(c);
  *med_ref = hb[0];
}

// ---------------------------------------------------------------------------
// Allocation-free background estimate (dgpu_estimate_background_noalloc): the
// launches of run_background, with the sample keys (at most 2^19 for any frame
// below 2^31 pixels: step = n / 2^18) and the two results in one fixed, file-scope
// device array instead of the context's workspace. The array is shared by every
// call on a device: calls that overlap in time (other streams or threads) race
// on it and must be serialised by the caller.
// ---------------------------------------------------------------------------
struct NoAllocBackground {
  float result[4];  // [0] median, [1] MAD
  uint32_t keys[kMedianMax];
};
static __device__ __align__(256) NoAllocBackground g_noalloc_background;

void background_noalloc(int64_t n, const float* img, const uint8_t* mask, cudaStream_t s, float* out2) {
  // Resolved on every call (a cheap lookup, no allocation) rather than cached:
  // after a device reset the runtime reloads the module and the array may sit at
  // a new address.
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_background);
  if (e != cudaSuccess)
    fail(DGPU_ERR_CUDA, std::string("estimate_background_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
  auto* sc = static_cast<NoAllocBackground*>(p);
  const float* res = sc->result;
  const MedianJob job = background_job(n, img, mask, sc->result);
  launch_medians(s, &job, 1, sc->keys);
  DGPU_CUDA(cudaMemcpyAsync(out2, res, 2 * sizeof(float), cudaMemcpyDeviceToHost, s));
  DGPU_CUDA(cudaStreamSynchronize(s));
}

}  // namespace dgpu
