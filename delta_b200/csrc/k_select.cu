// Radix-select sample medians (select_internal.h).
//
// Up to 2^19 values (every background sample, and the fill values of frames up
// to 3.6 Mpix): a cluster of eight CTAs per sample holds the keys in shared memory
// (the first 425984; each pass re-reads the rest, six loads in flight: one by one they
// made a pass over 523776 values 12 load latencies long) and selects without leaving
// it. A subsample of 512 keys first brackets the
// wanted rank (4 sigma of its rank: about a sixth of the keys), so that one
// pass of comparisons counts the keys below and only the bracket's keys enter the
// shared-memory histograms, spread over their digits; the leading bits of a sky
// background are all but constant, and histograms of them serialise on a few
// bins. A bracket that misses (it cannot for long on real samples) is replaced
// by the full range. Histograms are read by all eight CTAs through distributed
// shared memory after one cluster barrier, so every CTA picks the digit for
// itself. The MAD is a second select over |value - median| formed from the same
// keys. Samples of more than 2^16 values are gathered by a launch over the whole
// chip first (a strided value costs a 32-byte sector, which eight SMs draw
// slowly). With a launch per digit, a background took 13 launches and 75 us of
// device time; the two images of a pair (1003x1531, 2^18 values each) together
// take 2 launches and 42 us, the median and the MAD of each.
//
// More values: the gathering launch also brackets the median, a second one lists
// the bracket's keys, and the cluster finishes on the list.
// No host synchronisation anywhere: counts, ranks and brackets stay on the
// device.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "select_internal.h"

namespace cg = cooperative_groups;

namespace dgpu {

namespace {

constexpr int kCtas = 8;
constexpr int kThreads = 1024;
constexpr uint32_t kNone = 0xffffffffu;  // no finite value has this key, nor has any distance
constexpr int kSmemKeys = 52 * kThreads;  // keys a CTA holds at most (208 KB); the rest is re-read per pass
constexpr int kSub = 512;                // subsample
constexpr int kDigit = 10;               // bits per histogram
constexpr int kBins = 1 << kDigit;
static_assert(kBins == kThreads, "a bin per thread");
constexpr int64_t kDirect = int64_t(1) << 16;  // samples that the cluster gathers itself

// State of a large select.
struct BigSelect {
  unsigned arrived;   // blocks done gathering
  unsigned lo, hi;    // bracket of the median's key
  unsigned total;     // keys
  unsigned below;     // keys below lo
  unsigned listed;    // keys of [lo, hi] in the list
};

struct Jobs {
  MedianJob j[kMedianJobs];
  const uint32_t* keys[kMedianJobs] = {};  // gathered keys, else the sample is read
  const uint32_t* list = nullptr;          // large samples: the bracket's keys
  const BigSelect* big = nullptr;
};

__device__ __forceinline__ uint32_t sample_key(const MedianJob& j, int64_t at) {
  const int64_t i = at * j.step;
  const float x = __ldg(j.v + i);
  const uint8_t m = j.mask ? __ldg(j.mask + i) : 0;  // both loads in flight
  return isfinite(x) && m == 0 ? float_key(x) : kNone;
}

// Entry i of a subsample of m out of n entries: one of each n / m, at a place of its
// own (a fixed step can follow a frame's columns, e.g. its masked edge).
__device__ __forceinline__ int64_t sub_place(int i, int m, int64_t n) {
  const int64_t a = n * i / m, b = n * (i + 1) / m;
  const uint32_t h = static_cast<uint32_t>(i + 1) * 0x9e3779b1u;
  return min(n - 1, a + static_cast<int64_t>((static_cast<uint64_t>(h) * static_cast<uint64_t>(b - a)) >> 32));
}

// How many of the subsample's quads part, part + parts, ... are below k, and how many
// not above it.
__device__ __forceinline__ void count_around(const uint32_t* sub, int part, int parts, uint32_t k, int& less, int& upto) {
  less = upto = 0;
#pragma unroll 4
  for (int i = 4 * part; i < kSub; i += 4 * parts) {
    const uint4 q = *reinterpret_cast<const uint4*>(sub + i);
    less += (q.x < k) + (q.y < k) + (q.z < k) + (q.w < k);
    upto += (q.x <= k) + (q.y <= k) + (q.z <= k) + (q.w <= k);
  }
}

// The ranks [a, b] of the subsample that bracket rank fraction num / den of the
// sample; false where the subsample is too small to say. Any whole warp.
__device__ bool bracket_ranks(const uint32_t* sub, unsigned num, unsigned den, int& a, int& b) {
  int valid = 0;
  for (int i = threadIdx.x & 31; i < kSub; i += 32) valid += sub[i] != kNone;
  valid = __reduce_add_sync(0xffffffffu, valid);
  if (valid < 64 || den == 0) return false;
  const int at = min(valid - 1, static_cast<int>(static_cast<float>(valid) * (static_cast<float>(num) / static_cast<float>(den))));
  const int d = static_cast<int>(2.0f * sqrtf(static_cast<float>(valid))) + 2;
  a = max(0, at - d);
  b = min(valid - 1, at + d);
  return true;
}

__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kThreads, 1) k_cluster_median(Jobs jobs) {
  extern __shared__ __align__(16) uint32_t keys[];
  __shared__ __align__(16) uint32_t sub[kSub];
  __shared__ uint32_t mine[kSub / kCtas];
  __shared__ uint32_t bound[2];
  __shared__ unsigned hist[2][kBins];
  __shared__ unsigned cnt[2][2];  // this CTA's keys, and those below the bracket
  __shared__ unsigned sums[2];    // the cluster's
  __shared__ unsigned warp_n[32];
  __shared__ unsigned pick[2];    // digit, rank within it
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = static_cast<int>(cl.block_rank()), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ji = blockIdx.x / kCtas;
  const MedianJob j = jobs.j[ji];
  const int64_t sample = (j.n + j.step - 1) / j.step;
  // Large samples: the list, unless its bracket missed the median.
  bool listed = false;
  unsigned want_listed = 0;
  if (jobs.big) {
    const unsigned w = jobs.big->total / 2;
    listed = w >= jobs.big->below && w - jobs.big->below < jobs.big->listed;
    want_listed = w - jobs.big->below;
  }
  const uint32_t* src = listed ? jobs.list : jobs.keys[ji];
  const int64_t ns = listed ? jobs.big->listed : sample;
  const int64_t chunk = ((ns + kCtas - 1) / kCtas + 3) & ~int64_t(3), base = rank * chunk;
  const int count = static_cast<int>(max(static_cast<int64_t>(0), min(ns - base, chunk)));
  const int held = min(count, kSmemKeys), held4 = (held + 3) & ~3;
  if (rank == 0)
    for (int i = tid; i < j.nclear; i += kThreads) j.clear[i] = 0u;
  auto source = [&](int i) { return src ? __ldg(src + base + i) : sample_key(j, base + i); };
  if (src) {
#pragma unroll 4
    for (int i = 4 * tid; i + 3 < held; i += 4 * kThreads)
      *reinterpret_cast<uint4*>(keys + i) = __ldg(reinterpret_cast<const uint4*>(src + base + i));
    if (tid < 4 && (held & ~3) + tid < held4) keys[(held & ~3) + tid] = (held & ~3) + tid < held ? source((held & ~3) + tid) : kNone;
  } else {
#pragma unroll 4
    for (int i = tid; i < held4; i += kThreads) keys[i] = i < held ? source(i) : kNone;
  }
  for (int i = tid; i < kBins; i += kThreads) hist[0][i] = hist[1][i] = 0u;
  if (tid < 4) cnt[tid >> 1][tid & 1] = 0u;
  __syncthreads();
  int buf = 0;
  float med = 0.0f;
  auto distance = [&](uint32_t k) { return k == kNone ? k : float_key(fabsf(key_float(k) - med)); };
  for (int which = 0; which <= (j.mad ? 1 : 0); ++which) {
    if (which == 1) {
      for (int i = tid; i < held4; i += kThreads) keys[i] = distance(keys[i]);
      __syncthreads();
    }
    // f(key) over this CTA's keys, the held ones four at a time.
    auto each = [&](auto f) {
#pragma unroll 2
      for (int i = 4 * tid; i < held4; i += 4 * kThreads) {
        const uint4 q = *reinterpret_cast<const uint4*>(keys + i);
        f(q.x);
        f(q.y);
        f(q.z);
        f(q.w);
      }
      constexpr int kTail = 6;  // loads in flight (the largest sample's tail is 12 a thread)
      for (int i = held + tid; i < count; i += kTail * kThreads) {
        uint32_t k[kTail];
#pragma unroll
        for (int u = 0; u < kTail; ++u) k[u] = i + u * kThreads < count ? source(i + u * kThreads) : kNone;
#pragma unroll
        for (int u = 0; u < kTail; ++u) f(which == 1 ? distance(k[u]) : k[u]);
      }
    };
    if (tid < kSub / kCtas)
      mine[tid] = held > 0 ? keys[sub_place(tid, kSub / kCtas, held)] : kNone;
    if (tid == 0) {  // the full range, unless the subsample says better
      bound[0] = 0u;
      bound[1] = kNone - 1u;
    }
    cl.sync();
    for (int i = tid; i < kSub; i += kThreads)
      sub[i] = *cl.map_shared_rank(&mine[i % (kSub / kCtas)], i / (kSub / kCtas));
    __syncthreads();
    // This CTA ranks its own keys among all, 16 threads a key; the owner of a
    // bounding rank tells every CTA.
    int a, b;
    if (bracket_ranks(sub, listed ? want_listed : 1u, listed ? static_cast<unsigned>(ns) : 2u, a, b)) {
      constexpr int per = kThreads / (kSub / kCtas);
      const uint32_t k = mine[tid / per];
      int less, upto;
      count_around(sub, tid % per, per, k, less, upto);
      for (int o = 1; o < per; o <<= 1) {
        less += __shfl_xor_sync(0xffffffffu, less, o);
        upto += __shfl_xor_sync(0xffffffffu, upto, o);
      }
      if (tid % per < kCtas && k != kNone) {
        if (less <= a && a < upto) *cl.map_shared_rank(&bound[0], tid % per) = k;
        if (less <= b && b < upto) *cl.map_shared_rank(&bound[1], tid % per) = k;
      }
    }
    cl.sync();
    uint32_t lo = bound[0], hi = bound[1], result = 0u;
    bool empty = false;
    for (int attempt = 0; attempt < 2; ++attempt) {
      uint32_t prefix = 0u;
      unsigned want = 0u;
      bool missed = false;
      const uint32_t range = hi - lo;
      const int bits = 32 - __clz(range | 1u);
      for (int top = bits; top > 0 && !missed; top = max(top - kDigit, 0)) {
        const int shift = max(top - kDigit, 0);
        const unsigned mask = (1u << (top - shift)) - 1u;
        if (top == bits) {
          unsigned n_all = 0, n_below = 0;
          each([&](uint32_t k) {
            n_all += k != kNone;
            n_below += k < lo;
            const uint32_t d = k - lo;
            if (k >= lo && d <= range) atomicAdd(&hist[buf][d >> shift], 1u);
          });
          n_all = __reduce_add_sync(0xffffffffu, n_all);
          n_below = __reduce_add_sync(0xffffffffu, n_below);
          if (lane == 0) {
            atomicAdd(&cnt[buf][0], n_all);
            atomicAdd(&cnt[buf][1], n_below);
          }
        } else {
          const uint32_t at = prefix >> top;
          each([&](uint32_t k) {
            const uint32_t d = k - lo;
            if (k >= lo && d <= range && (d >> top) == at) atomicAdd(&hist[buf][(d >> shift) & mask], 1u);
          });
        }
        cl.sync();  // every CTA's histogram is complete (and the other buffer is read)
        unsigned h = 0;  // kBins == kThreads: a bin per thread
#pragma unroll
        for (int r = 0; r < kCtas; ++r) h += *cl.map_shared_rank(&hist[buf][tid], r);
        hist[buf ^ 1][tid] = 0u;
        if (tid < 2) {
          unsigned s = 0;
#pragma unroll
          for (int r = 0; r < kCtas; ++r) s += *cl.map_shared_rank(&cnt[buf][tid], r);
          sums[tid] = s;
          cnt[buf ^ 1][tid] = 0u;
          pick[0] = kNone;  // stays where the rank lies past the bracket
        }
        unsigned incl = h;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        if (lane == 31) warp_n[warp] = incl;
        __syncthreads();
        unsigned before = lane < warp ? warp_n[lane] : 0u;
        before = __reduce_add_sync(0xffffffffu, before);
        if (top == bits) {
          const unsigned w = listed ? want_listed : sums[0] / 2;
          empty = sums[0] == 0;
          missed = w < sums[1];
          want = w - sums[1];
        }
        const unsigned excl = before + incl - h;
        if (!missed && want >= excl && want - excl < h) {
          pick[0] = static_cast<unsigned>(tid);
          pick[1] = want - excl;
        }
        __syncthreads();
        buf ^= 1;
        if (pick[0] == kNone) missed = true;
        if (!missed) {
          prefix |= pick[0] << shift;
          want = pick[1];
        }
        __syncthreads();  // pick, sums and warp_n are rewritten
      }
      result = lo + prefix;
      if (empty || !missed) break;
      lo = 0u;
      hi = kNone - 1u;
    }
    med = empty ? 0.0f : key_float(result);
    if (rank == 0 && tid == 0) j.out[which] = med;
  }
  cl.sync();  // no CTA leaves while another reads its shared memory
}

// Keys of up to two samples, over the whole chip. With `big` (one sample) the
// last block brackets the median from a subsample.
__global__ void __launch_bounds__(256) k_gather_keys(Jobs jobs, uint32_t* keys0, uint32_t* keys1, BigSelect* big) {
  __shared__ __align__(16) uint32_t sub[kSub];
  __shared__ bool last;
  const MedianJob j = jobs.j[blockIdx.y];
  uint32_t* keys = blockIdx.y ? keys1 : keys0;
  const int tid = threadIdx.x;
  const int64_t ns = (j.n + j.step - 1) / j.step;
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * 2048; b < ns; b += static_cast<int64_t>(gridDim.x) * 2048) {
    uint32_t k[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t at = b + u * 256 + tid;
      k[u] = at < ns ? sample_key(j, at) : kNone;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t at = b + u * 256 + tid;
      if (at < ns) keys[at] = k[u];
    }
  }
  if (big == nullptr) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&big->arrived, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = tid; i < kSub; i += 256) sub[i] = __ldcg(keys + sub_place(i, kSub, ns));
  __syncthreads();
  if (tid == 0) {
    big->lo = 0u;
    big->hi = kNone - 1u;
  }
  __syncthreads();
  int a, b;
  if (!bracket_ranks(sub, 1u, 2u, a, b)) return;
  for (int e = tid; e < kSub; e += 256) {
    const uint32_t k = sub[e];
    int less, upto;
    count_around(sub, 0, 1, k, less, upto);
    if (k == kNone) continue;
    if (less <= a && a < upto) big->lo = k;
    if (less <= b && b < upto) big->hi = k;
  }
}

// The bracket's keys (in any order: only their multiset counts), and how many
// keys there are and lie below it.
__global__ void __launch_bounds__(256) k_list_bracket(int64_t ns, const uint32_t* __restrict__ keys, BigSelect* big,
                                                      uint32_t* __restrict__ list) {
  __shared__ unsigned warp_n[8];
  __shared__ unsigned at, sums[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lo = big->lo, hi = big->hi;
  if (tid < 2) sums[tid] = 0u;
  unsigned n_all = 0, n_below = 0;
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * 2048; b < ns; b += static_cast<int64_t>(gridDim.x) * 2048) {
    uint32_t k[8];
    unsigned in = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t i = b + u * 256 + tid;
      k[u] = i < ns ? __ldg(keys + i) : kNone;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      n_all += k[u] != kNone;
      n_below += k[u] < lo;
      if (k[u] >= lo && k[u] <= hi) in |= 1u << u;
    }
    const unsigned own = __popc(in);
    unsigned incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_n[warp] = incl;
    __syncthreads();
    if (tid == 0) {
      unsigned t = 0;
      for (int i = 0; i < 8; ++i) {
        const unsigned c = warp_n[i];
        warp_n[i] = t;
        t += c;
      }
      at = t ? atomicAdd(&big->listed, t) : 0u;
    }
    __syncthreads();
    unsigned o = at + warp_n[warp] + incl - own;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (in & (1u << u)) list[o++] = k[u];
    __syncthreads();
  }
  n_all = __reduce_add_sync(0xffffffffu, n_all);
  n_below = __reduce_add_sync(0xffffffffu, n_below);
  if (lane == 0) {
    atomicAdd(&sums[0], n_all);
    atomicAdd(&sums[1], n_below);
  }
  __syncthreads();
  if (tid == 0) {
    if (sums[0]) atomicAdd(&big->total, sums[0]);
    if (sums[1]) atomicAdd(&big->below, sums[1]);
  }
}

int gather_blocks(int64_t ns) { return static_cast<int>(std::min<int64_t>((ns + 2047) / 2048, 148 * 4)); }

void launch_cluster(cudaStream_t s, const Jobs& jobs, int njobs, int64_t most) {
  const int64_t held = std::min<int64_t>(((most + kCtas - 1) / kCtas + 3) & ~int64_t(3), kSmemKeys);
  const size_t smem = sizeof(uint32_t) * static_cast<size_t>(std::max<int64_t>(held, 4));
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_cluster_median), smem);
  k_cluster_median<<<kCtas * njobs, kThreads, smem, s>>>(jobs);
  DGPU_LAUNCH("k_cluster_median");
}

int64_t sample_size(const MedianJob& j) { return (j.n + j.step - 1) / j.step; }

}  // namespace

size_t medians_scratch(const MedianJob* jobs, int njobs) {
  int64_t n = 0;
  for (int i = 0; i < njobs; ++i) n += (sample_size(jobs[i]) + 3) & ~int64_t(3);  // 16-byte aligned samples
  return sizeof(uint32_t) * static_cast<size_t>(n);
}

void launch_medians(cudaStream_t s, const MedianJob* jobs, int njobs, void* scratch) {
  Jobs js;
  int64_t most = 0;
  for (int i = 0; i < njobs; ++i) {
    js.j[i] = jobs[i];
    most = std::max(most, sample_size(jobs[i]));
  }
  if (most > kMedianMax) fail(DGPU_ERR_INVALID, "median: sample too large");
  if (most > kDirect) {
    uint32_t* keys0 = static_cast<uint32_t*>(scratch);
    uint32_t* keys1 = keys0 + ((sample_size(jobs[0]) + 3) & ~int64_t(3));
    k_gather_keys<<<dim3(gather_blocks(most), njobs), 256, 0, s>>>(js, keys0, keys1, nullptr);
    DGPU_LAUNCH("k_gather_keys");
    js.keys[0] = keys0;
    js.keys[1] = keys1;
  }
  launch_cluster(s, js, njobs, most);
}

void launch_upper_median(Context& c, int64_t n, int64_t step, const float* v, const uint8_t* mask, float* out) {
  MedianJob j;
  j.v = v;
  j.mask = mask;
  j.n = n;
  j.step = step;
  j.out = out;
  const int64_t ns = sample_size(j);
  auto* keys = static_cast<uint32_t*>(c.slot(kSlotSamples, (ns > kMedianMax ? 2 : 1) * medians_scratch(&j, 1)));
  if (ns <= kMedianMax) {
    launch_medians(c.stream, &j, 1, keys);
    return;
  }
  auto* big = static_cast<BigSelect*>(c.slot(kSlotSelect, sizeof(BigSelect)));
  uint32_t* list = keys + ((ns + 3) & ~int64_t(3));
  Jobs js;
  js.j[0] = j;
  js.keys[0] = keys;
  js.list = list;
  js.big = big;
  DGPU_CUDA(cudaMemsetAsync(big, 0, sizeof(BigSelect), c.stream));
  k_gather_keys<<<gather_blocks(ns), 256, 0, c.stream>>>(js, keys, keys, big);
  DGPU_LAUNCH("k_gather_keys");
  k_list_bracket<<<gather_blocks(ns), 256, 0, c.stream>>>(ns, keys, big, list);
  DGPU_LAUNCH("k_list_bracket");
  launch_cluster(c.stream, js, 1, kMedianMax);
}

}  // namespace dgpu
