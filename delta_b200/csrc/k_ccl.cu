// Connected-component source catalog (src/catalog.cpp:61-697) on sm_100a.
//
// Seeds are rare (a few thousand of 1.7e7 pixels), so one pass over the score and
// mask packs both polarities into bitmaps and everything after it works on the
// raster-ordered list of the wanted polarity's seed pixels: 8-connected
// union-find over list positions with atomicMin linking (every parent is below
// its child, so each component's root is its first pixel in raster order) ->
// roots ranked in list order, which reproduces the reference's final numbering
// exactly (label = rank of the component's first pixel in raster order,
// src/catalog.cpp:124-260) -> per-label reductions with atomics (count,
// |score|-weighted sums in FP64, peak with the lowest-index tie-break of
// src/catalog.cpp:362-371, mask OR over footprint + 8-ring, dipole contact) ->
// per-component finishing (centroid, FWHM consistency, aperture flux, quality
// bits, dipole flag, optional PSF-shape fit and bright-star distance). A
// neighbour's list position is the number of seeds before its bitmap word plus
// the set bits below its own. The label image itself is written only where it
// is asked for (expand_labels). Every data-dependent loop is capped; hitting a
// cap sets the context status word and the call reports DGPU_ERR_LIMIT.
// Floor at 4096^2: reading 5 bytes a pixel, 13 us at 6.5 TB/s.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "dev_common.cuh"

namespace dgpu {


constexpr int kSeedBlock = 8192;  // pixels per block of the seed pass
constexpr int kRankBlock = 1024;  // list entries per block of the ranking
static_assert(kSeedBlock == 8 * 8 * 128, "eight warps of eight groups of 128 pixels");

// The catalog's work arrays, sized for every pixel a seed: bitmaps of the
// labelled polarity and the other one, the number of listed seeds before each
// word, the seed list, the union-find parents (list positions), the rank of each
// root, per-block counts of the seed pass and of the ranking, and
// {arrival counters (2), seeds, roots}.
struct SeedList {
  unsigned* bits;
  unsigned* other;
  int* before;
  int* list;
  int* parent;
  int* rank;
  int* seed_counts;
  int* root_counts;
  int* heads;  // [0], [1]: blocks arrived; [2]: seeds; [3]: roots

  static int64_t words(int64_t n) { return (n + 31) / 32; }
  static int64_t blocks(int64_t n) { return (n + kSeedBlock - 1) / kSeedBlock; }
  static int64_t ranks(int64_t n) { return (n + kRankBlock - 1) / kRankBlock; }
  static size_t ints(int64_t n) {
    return static_cast<size_t>(3 * words(n) + 3 * n + blocks(n) + ranks(n)) + 4;
  }
  static SeedList at(int* p, int64_t n) {
    SeedList l;
    l.heads = p;
    l.bits = reinterpret_cast<unsigned*>(p + 4);
    l.other = l.bits + words(n);
    l.before = reinterpret_cast<int*>(l.other + words(n));
    l.list = l.before + words(n);
    l.parent = l.list + n;
    l.rank = l.parent + n;
    l.seed_counts = l.rank + n;
    l.root_counts = l.seed_counts + blocks(n);
    return l;
  }
};

// Exclusive scan of counts[0 .. nb) in place by one block of 256 threads;
// returns the total to every thread.
__device__ int block_scan(int* counts, int nb) {
  __shared__ int part[8];
  __shared__ int total;
  const int per = (nb + 255) / 256, lo = min(nb, static_cast<int>(threadIdx.x) * per), hi = min(nb, lo + per);
  int s = 0;
#pragma unroll 8
  for (int i = lo; i < hi; ++i) s += __ldcg(counts + i);
  int v = s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) part[warp] = v;
  __syncthreads();
  int run = v - s;
  for (int i = 0; i < warp; ++i) run += part[i];
  if (threadIdx.x == 255) total = run + s;
  for (int i = lo; i < hi; ++i) {
    const int c = __ldcg(counts + i);
    counts[i] = run;
    run += c;
  }
  __syncthreads();
  return total;
}

// Does this block arrive last? (Every block's writes before the call are then
// visible to it; no block waits for another.)
__device__ bool last_block(int* arrived) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(arrived, 1) == static_cast<int>(gridDim.x) - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Bits 0-7 of x to every fourth bit.
__device__ __forceinline__ unsigned spread4(unsigned x) {
  x = (x | (x << 12)) & 0x000f000fu;
  x = (x | (x << 6)) & 0x03030303u;
  return (x | (x << 3)) & 0x11111111u;
}

// Bitmaps of both polarities and the labelled one's count per block; the last
// block scans the counts. A lane takes four adjacent pixels of each group of 128
// (one 16-byte and one 4-byte load where `vec` says that the images are aligned
// for it), all eight groups of its warp in flight.
__global__ void __launch_bounds__(256)
k_seed_bits(int64_t n, int nb, const float* __restrict__ score, const uint8_t* __restrict__ mask, bool vec,
            float thr_pos, float thr_neg, bool negative, SeedList sl) {
  __shared__ int wc[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kSeedBlock + warp * 1024 + 4 * lane;
  float v[8][4];
  unsigned m[8];  // a byte per pixel, non-zero: excluded
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const int64_t i = base + 128 * g;
    if (vec && i + 3 < n) {
      const float4 t = __ldcs(reinterpret_cast<const float4*>(score + i));
      v[g][0] = t.x, v[g][1] = t.y, v[g][2] = t.z, v[g][3] = t.w;
      m[g] = mask != nullptr ? __ldcs(reinterpret_cast<const unsigned*>(mask + i)) : 0u;
    } else {
      m[g] = 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        v[g][u] = i + u < n ? __ldcs(score + i + u) : __int_as_float(0x7fc00000);
        if (mask != nullptr && i + u < n) m[g] |= static_cast<unsigned>(__ldcs(mask + i + u)) << (8 * u);
      }
    }
  }
  int count = 0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    unsigned p[4], q[4];  // one bit per lane, by pixel of the four
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool good = isfinite(v[g][u]) && ((m[g] >> (8 * u)) & 0xffu) == 0;
      p[u] = __ballot_sync(0xffffffffu, good && v[g][u] >= thr_pos);
      q[u] = __ballot_sync(0xffffffffu, good && v[g][u] <= -thr_neg);
    }
    // Word `lane` (0-3) of the group: pixel 4 k + u of it is bit k of byte `lane` of ballot u.
    const int64_t i = base - 4 * lane + 128 * g + 32 * lane;
    if (lane < 4 && i < n) {
      unsigned pw = 0, qw = 0;
      if (p[0] | p[1] | p[2] | p[3] | q[0] | q[1] | q[2] | q[3])
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          pw |= spread4((p[u] >> (8 * lane)) & 0xffu) << u;
          qw |= spread4((q[u] >> (8 * lane)) & 0xffu) << u;
        }
      sl.bits[i >> 5] = negative ? qw : pw;
      sl.other[i >> 5] = negative ? pw : qw;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) count += __popc(negative ? q[u] : p[u]);
  }
  if (lane == 0) wc[warp] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < 8; ++i) t += wc[i];
    sl.seed_counts[blockIdx.x] = t;
  }
  if (last_block(&sl.heads[0])) {
    const int total = block_scan(sl.seed_counts, nb);
    if (threadIdx.x == 0) sl.heads[2] = total;
  }
}

// The seed list in raster order, each seed its own parent.
__global__ void __launch_bounds__(kSeedBlock / 32)
k_seed_list(int64_t n, int nb, SeedList sl) {
  const int b = blockIdx.x;
  const int at0 = sl.seed_counts[b], at1 = b + 1 < nb ? sl.seed_counts[b + 1] : sl.heads[2];
  if (at0 == at1) return;
  __shared__ int wt[kSeedBlock / 32 / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t word = static_cast<int64_t>(b) * (kSeedBlock / 32) + threadIdx.x;
  unsigned bits = word * 32 < n ? sl.bits[word] : 0u;
  int v = __popc(bits);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) wt[warp] = v;
  __syncthreads();
  int at = at0 + v - __popc(bits);
  for (int i = 0; i < warp; ++i) at += wt[i];
  if (word * 32 < n) sl.before[word] = at;
  while (bits) {
    sl.list[at] = static_cast<int>(word * 32) + __ffs(bits) - 1;
    sl.parent[at] = at;
    ++at;
    bits &= bits - 1;
  }
}

__device__ __forceinline__ bool has_bit(const unsigned* bits, int i) { return (bits[i >> 5] >> (i & 31)) & 1u; }
__device__ __forceinline__ int list_pos(const SeedList& sl, int i) {
  return sl.before[i >> 5] + __popc(sl.bits[i >> 5] & ((1u << (i & 31)) - 1u));
}

__device__ __forceinline__ int find_root(const int* L, int i, unsigned* st, int cap) {
  for (int it = 0; it < cap; ++it) {
    const int p = L[i];
    if (p == i) return i;
    i = p;
  }
  set_status(st, kStatusLoopLimit);
  return i;
}

__device__ void unite(int* L, int a, int b, unsigned* st, int cap) {
  for (int it = 0; it < cap; ++it) {
    a = find_root(L, a, st, cap);
    b = find_root(L, b, st, cap);
    if (a == b) return;
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&L[a], b);
    if (old == a) return;
    a = old;
  }
  set_status(st, kStatusLoopLimit);
}

__global__ void k_label_merge(int w, SeedList sl, unsigned* st, int cap) {
  const int n = sl.heads[2];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int i = sl.list[e], x = i % w;
    if (x > 0 && has_bit(sl.bits, i - 1)) unite(sl.parent, e, e - 1, st, cap);
    if (i >= w) {
      const int a = i - w;
      if (x > 0 && has_bit(sl.bits, a - 1)) unite(sl.parent, e, list_pos(sl, a - 1), st, cap);
      if (has_bit(sl.bits, a)) unite(sl.parent, e, list_pos(sl, a), st, cap);
      if (x + 1 < w && has_bit(sl.bits, a + 1)) unite(sl.parent, e, list_pos(sl, a + 1), st, cap);
    }
  }
}

// Parents to roots; the roots of each block of list entries are counted and the
// last block scans the counts.
__global__ void __launch_bounds__(256) k_label_flatten(SeedList sl, unsigned* st, int cap) {
  __shared__ int wc[8];
  const int n = sl.heads[2], nb = (n + kRankBlock - 1) / kRankBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    int count = 0;
    for (int e0 = b * kRankBlock + warp * 128; e0 < b * kRankBlock + (warp + 1) * 128; e0 += 32) {
      const int e = e0 + lane;
      int r = -1;
      if (e < n) {
        r = find_root(sl.parent, e, st, cap);
        sl.parent[e] = r;
      }
      count += __popc(__ballot_sync(0xffffffffu, e < n && r == e));
    }
    if (lane == 0) wc[warp] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int i = 0; i < 8; ++i) t += wc[i];
      sl.root_counts[b] = t;
    }
    __syncthreads();
  }
  if (last_block(&sl.heads[1])) {
    const int total = block_scan(sl.root_counts, nb);
    if (threadIdx.x == 0) sl.heads[3] = total;
  }
}

// rank[root] = raster rank of the root (0-based).
__global__ void __launch_bounds__(256) k_root_rank(SeedList sl) {
  __shared__ int wc[8];
  const int n = sl.heads[2], nb = (n + kRankBlock - 1) / kRankBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    unsigned roots[4];
    int count = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int e = b * kRankBlock + warp * 128 + g * 32 + lane;
      roots[g] = __ballot_sync(0xffffffffu, e < n && sl.parent[e] == e);
      count += __popc(roots[g]);
    }
    __syncthreads();
    if (lane == 0) wc[warp] = count;
    __syncthreads();
    int at = sl.root_counts[b];
    for (int i = 0; i < warp; ++i) at += wc[i];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int e = b * kRankBlock + warp * 128 + g * 32 + lane;
      if (roots[g] & (1u << lane)) sl.rank[e] = at + __popc(roots[g] & ((1u << lane) - 1u));
      at += __popc(roots[g]);
    }
  }
}

// Component (label - 1) of list entry e. Only a root carries a rank, so an entry
// maps to a component only through a root: one left pointing at a non-root (a
// capped search gave up) gets -1 and the bounds status, which keeps every
// component within [0, number of roots).
__device__ __forceinline__ int component_of(const SeedList& sl, int e, unsigned* st) {
  const int r = sl.parent[e];
  if (sl.parent[r] == r) return sl.rank[r];
  set_status(st, kStatusBounds);
  return -1;
}

// The label image: zeros, then label = component + 1 at the seeds.
__global__ void k_expand_labels(SeedList sl, int* __restrict__ labels, unsigned* st) {
  const int n = sl.heads[2];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    labels[sl.list[e]] = component_of(sl, e, st) + 1;
}

// Per-component accumulators (index label-1).
struct CompStats {
  int* count;
  double* sum;
  double* sx;
  double* sy;
  unsigned long long* peak;  // (bits(|score|) << 32) | ~idx -> max gives lowest idx on ties
  unsigned* mask_or;
  unsigned* touched;
  int* first;  // minimum linear index (the root)
};

// Reductions of every seed into its component. A seed's 8-neighbours of the same
// polarity are in its own component, so the mask ring takes the neighbours that
// are not seeds; a neighbour (or the pixel itself) carrying the other polarity
// marks the component (flag_dipole_positives, src/catalog.cpp:431-458).
__global__ void k_comp_reduce(int w, int h, SeedList sl, const float* __restrict__ score,
                              const uint8_t* __restrict__ mask, CompStats cs, unsigned* st) {
  const int n = sl.heads[2];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int c = component_of(sl, e, st);
    if (c < 0) continue;
    const int i = sl.list[e], x = i % w, y = i / w;
    const double wt = fabs(static_cast<double>(score[i]));
    atomicAdd(&cs.count[c], 1);
    atomicAdd(&cs.sum[c], wt);
    atomicAdd(&cs.sx[c], wt * x);
    atomicAdd(&cs.sy[c], wt * y);
    const unsigned long long key =
        (static_cast<unsigned long long>(__float_as_uint(fabsf(score[i]))) << 32) |
        static_cast<unsigned long long>(0xffffffffu - static_cast<unsigned>(i));
    atomicMax(&cs.peak[c], key);
    atomicMin(&cs.first[c], i);
    unsigned m = mask ? mask[i] : 0u;
    bool touched = false;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        if (y + dy < 0 || y + dy >= h || x + dx < 0 || x + dx >= w) continue;
        const int j = i + dy * w + dx;
        touched = touched || has_bit(sl.other, j);
        if (mask && !has_bit(sl.bits, j)) m |= mask[j];
      }
    if (m) atomicOr(&cs.mask_or[c], m);
    if (touched) cs.touched[c] = 1u;
  }
}

struct CompOut {
  double* x;
  double* y;
  int* peak_x;
  int* peak_y;
  double* peak_snr;
  int* n_pix;
  double* flux;
  double* expected_n_pix;
  double* fwhm_ratio;
  uint8_t* fwhm_consistent;
  uint8_t* mask_flags;
  uint8_t* is_dipole;
  uint8_t* quality;
  double* psf_chi2;
  int* psf_chi2_dof;
  double* psf_amplitude;
  double* psf_amplitude_err;
  uint8_t* shape_consistent;
  double* bright_star_dist;
  uint8_t* near_bright_star;
};

struct FinishParams {
  double threshold;  // the seeding threshold of this polarity
  double expected_fwhm, tol_lo, tol_hi;
  int aperture_radius;
  int do_shape, do_bright;
  double shape_tol, bright_radius;
  int psf_size;
};

__device__ long lround_away(double v) { return static_cast<long>(v >= 0 ? floor(v + 0.5) : -floor(-v + 0.5)); }

// summarize_component (src/catalog.cpp:337-418) finishing + dipole flag +
// enrich_entries (src/catalog.cpp:476-596). WARP: a warp per component, its lanes load
// the aperture's pixels together and every lane adds them in raster order; else a
// thread per component.
template <bool WARP>
__global__ void __launch_bounds__(128) k_comp_finish(int ncomp, int w, int h, const float* __restrict__ score,
                              const float* __restrict__ diff, const uint8_t* __restrict__ mask,
                              const float* __restrict__ variance, const float* __restrict__ psf,
                              const double* __restrict__ bx, const double* __restrict__ by, int nb,
                              CompStats cs, FinishParams fp, CompOut o) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, c = WARP ? t >> 5 : t, lane = threadIdx.x & 31;
  if (c >= ncomp) return;
  const double kFwhmPerSigma = 2.354820045030949;
  const double kPi = 3.14159265358979323846;
  const int cnt = cs.count[c];
  const double sum = cs.sum[c];
  const int first = cs.first[c];
  double x = sum > 0.0 ? cs.sx[c] / sum : static_cast<double>(first % w);
  double y = sum > 0.0 ? cs.sy[c] / sum : static_cast<double>(first / w);
  const unsigned long long pk = cs.peak[c];
  const int pidx = static_cast<int>(0xffffffffu - static_cast<unsigned>(pk & 0xffffffffull));
  const double peak_snr = static_cast<double>(score[pidx]);
  o.x[c] = x;
  o.y[c] = y;
  o.peak_x[c] = pidx % w;
  o.peak_y[c] = pidx / w;
  o.peak_snr[c] = peak_snr;
  o.n_pix[c] = cnt;
  const unsigned mflags = cs.mask_or[c] & 0xffu;
  o.mask_flags[c] = static_cast<uint8_t>(mflags);
  const double sigma = fp.expected_fwhm / kFwhmPerSigma;
  const double ratio = fp.threshold > 0.0 ? fabs(peak_snr) / fp.threshold : 0.0;
  const double log_term = ratio > 0.0 ? log(ratio * ratio) : 0.0;
  const double expn = kPi * sigma * sigma * fmax(0.0, log_term);
  const double fr = expn > 0.0 ? cnt / expn : INFINITY;
  const bool consistent = fr >= fp.tol_lo && fr <= fp.tol_hi;
  o.expected_n_pix[c] = expn;
  o.fwhm_ratio[c] = fr;
  o.fwhm_consistent[c] = consistent ? 1 : 0;
  const int radius = fp.aperture_radius > 0 ? fp.aperture_radius
                                            : max(1, static_cast<int>(lround_away(3.0 * sigma)));
  {
    const int x0 = static_cast<int>(lround_away(x)), y0 = static_cast<int>(lround_away(y));
    const double r2 = static_cast<double>(radius) * radius;
    const int64_t side = 2 * static_cast<int64_t>(radius) + 1, area = side * side;
    double fsum = 0.0;
    if constexpr (WARP) {
      for (int64_t e0 = 0; e0 < area; e0 += 32) {
        const int64_t e = e0 + lane;
        const int dy = static_cast<int>(e / side) - radius, dx = static_cast<int>(e % side) - radius;
        const int yy = y0 + dy, xx = x0 + dx;
        float v = 0.0f;
        if (e < area && yy >= 0 && yy < h && xx >= 0 && xx < w && !(dx * dx + dy * dy > r2))
          v = diff[static_cast<int64_t>(yy) * w + xx];
        const unsigned in = __ballot_sync(0xffffffffu, v != 0.0f && isfinite(v));  // adding a zero changes nothing
        for (unsigned left = in; left; left &= left - 1)
          fsum += static_cast<double>(__shfl_sync(0xffffffffu, v, __ffs(left) - 1));
      }
    } else {
      for (int dy = max(-radius, -y0); dy <= min(radius, h - 1 - y0); ++dy)
        for (int dx = max(-radius, -x0); dx <= min(radius, w - 1 - x0); ++dx) {
          if (dx * dx + dy * dy > r2) continue;
          const float v = diff[static_cast<int64_t>(y0 + dy) * w + x0 + dx];
          if (isfinite(v)) fsum += static_cast<double>(v);
        }
    }
    o.flux[c] = fsum;
  }
  if (WARP && lane != 0) return;
  uint8_t q = 0;
  if (!consistent) q |= 1u;
  if (mflags != 0) q |= 4u;
  const bool dip = cs.touched[c] != 0;
  o.is_dipole[c] = dip ? 1 : 0;
  if (dip) q |= 2u;
  o.psf_chi2[c] = 0.0;
  o.psf_chi2_dof[c] = 0;
  o.psf_amplitude[c] = 0.0;
  o.psf_amplitude_err[c] = 0.0;
  o.shape_consistent[c] = 1;
  o.bright_star_dist[c] = INFINITY;
  o.near_bright_star[c] = 0;
  if (fp.do_shape) {
    const int ps = fp.psf_size, r = ps / 2;
    const int x0 = static_cast<int>(lround_away(x)), y0 = static_cast<int>(lround_away(y));
    double swdp = 0.0, swpp = 0.0;
    int used = 0;
    for (int pass = 0; pass < 2; ++pass) {
      double amp = pass ? swdp / swpp : 0.0;
      double chi2 = 0.0;
      for (int dy = -r; dy <= r; ++dy) {
        const int yy = y0 + dy;
        if (yy < 0 || yy >= h) continue;
        for (int dx = -r; dx <= r; ++dx) {
          const int xx = x0 + dx;
          if (xx < 0 || xx >= w) continue;
          const int64_t idx = static_cast<int64_t>(yy) * w + xx;
          if (mask && mask[idx] != 0) continue;
          const float v = variance[idx];
          const float d = diff[idx];
          if (!(v > 0.0f) || !isfinite(v) || !isfinite(d)) continue;
          const float p = psf[(dy + r) * ps + (dx + r)];
          if (pass == 0) {
            const double wgt = 1.0 / static_cast<double>(v);
            swdp += wgt * static_cast<double>(d) * p;
            swpp += wgt * static_cast<double>(p) * p;
            ++used;
          } else {
            const double res = static_cast<double>(d) - amp * static_cast<double>(p);
            chi2 += res * res / static_cast<double>(v);
          }
        }
      }
      if (pass == 0 && (used < 3 || !(swpp > 0.0))) break;
      if (pass == 1) {
        o.psf_amplitude[c] = amp;
        o.psf_amplitude_err[c] = sqrt(1.0 / swpp);
        o.psf_chi2[c] = chi2;
        o.psf_chi2_dof[c] = used - 1;
        const bool sc = (used - 1) > 0 ? (chi2 / (used - 1) <= fp.shape_tol) : true;
        o.shape_consistent[c] = sc ? 1 : 0;
        if (!sc) q |= 8u;
      }
    }
  }
  if (fp.do_bright) {
    double best2 = INFINITY;
    for (int i = 0; i < nb; ++i) {
      const double dx = x - bx[i], dy = y - by[i];
      const double d2 = dx * dx + dy * dy;
      if (d2 < best2) best2 = d2;
    }
    const double dist = sqrt(best2);
    o.bright_star_dist[c] = dist;
    const bool near = dist <= fp.bright_radius;
    o.near_bright_star[c] = near ? 1 : 0;
    if (near) q |= 16u;
  }
  o.quality[c] = q;
}

// ---------------------------------------------------------------------------
// Host driver
// ---------------------------------------------------------------------------

// Blocks of the kernels that walk the seed list (its length is on the device): as many
// as the chip holds, twice for the merge, whose searches take uneven time. Two blocks
// an SM save 1 us on a list of a few thousand and lose on long ones (4096 x 4096 of
// noise, threshold 0.3 sigma, 6e6 seeds: merge 1729 us, now 414; a comb of one
// component with 2e6 seeds 1649, now 366).
constexpr int kListBlocks = 148 * 8;
constexpr int kMergeBlocks = 148 * 16;
// Components that get a warp each for their finish: half the chip's warps. 4096 x 4096,
// a warp and a thread each: 66 components 10 and 18 us, 4100 15 and 26, 22933 57 and 28,
// 348091 776 and 68; 1001 x 1001: 1360 10 and 19, 6152 20 and 19.
constexpr int kFinishWarps = 148 * 32;

void expand_labels(Context& c, int64_t n, int* labels) {
  const SeedList sl = SeedList::at(static_cast<int*>(c.slot_ptr[kSlotLabels]), n);
  DGPU_CUDA(cudaMemsetAsync(labels, 0, sizeof(int) * n, c.stream));
  k_expand_labels<<<kListBlocks, 256, 0, c.stream>>>(sl, labels, c.d_status);
  DGPU_LAUNCH("k_expand_labels");
}

int run_catalog(Context& c, int w, int h, const float* score, const float* diff, const uint8_t* mask,
                const dgpu_catalog_params& p, const float* variance, const float* psf, int psf_size,
                const double* bright_x, const double* bright_y, int n_bright) {
  cudaStream_t s = c.stream;
  const int64_t n = static_cast<int64_t>(w) * h;
  // Until the list is complete there is nothing expand_labels could read: its indices
  // come from the list, which the work below overwrites.
  c.cat_npix = -1;
  c.cat_count = 0;
  const SeedList sl = SeedList::at(static_cast<int*>(c.slot(kSlotLabels, sizeof(int) * SeedList::ints(n))), n);
  const bool neg = p.return_negative != 0;
  const int nb = static_cast<int>(SeedList::blocks(n));
  {
    StageTimer t(c, "catalog: seed");
    DGPU_CUDA(cudaMemsetAsync(sl.heads, 0, sizeof(int) * 4, s));
    const uint8_t* excluded = p.exclude_bad_pixels ? mask : nullptr;
    const bool vec = reinterpret_cast<uintptr_t>(score) % 16 == 0 && reinterpret_cast<uintptr_t>(excluded) % 4 == 0;
    k_seed_bits<<<nb, 256, 0, s>>>(n, nb, score, excluded, vec,
                                   static_cast<float>(p.threshold_sigma),
                                   static_cast<float>(p.threshold_sigma_dipole), neg, sl);
    DGPU_LAUNCH("k_seed_bits");
  }
  int ncomp = 0;
  {
    StageTimer t(c, neg ? "catalog: label negative" : "catalog: label positive");
    k_seed_list<<<nb, kSeedBlock / 32, 0, s>>>(n, nb, sl);
    DGPU_LAUNCH("k_seed_list");
    k_label_merge<<<kMergeBlocks, 256, 0, s>>>(w, sl, c.d_status, c.label_loop_cap);
    DGPU_LAUNCH("k_label_merge");
    k_label_flatten<<<kListBlocks, 256, 0, s>>>(sl, c.d_status, c.label_loop_cap);
    DGPU_LAUNCH("k_label_flatten");
    k_root_rank<<<kListBlocks, 256, 0, s>>>(sl);
    DGPU_LAUNCH("k_root_rank");
    read_back(c, &ncomp, sl.heads + 3, sizeof(int));
    sync_reads(c);
  }
  c.cat_npix = n;
  c.cat_count = ncomp;
  c.cat_d.assign(static_cast<size_t>(ncomp) * 12, 0.0);
  c.cat_i.assign(static_cast<size_t>(ncomp) * 4, 0);
  c.cat_u8.assign(static_cast<size_t>(ncomp) * 8, 0);
  if (ncomp == 0) return 0;

  StageTimer t(c, neg ? "catalog: summarize negative" : "catalog: summarize positive");
  // Stats arrays in one slot.
  const size_t nc = static_cast<size_t>(ncomp);
  const size_t stats_bytes = nc * (4 + 8 * 3 + 8 + 4 + 4 + 4) + 256;
  char* sb = static_cast<char*>(c.slot(kSlotCompStats, stats_bytes));
  CompStats cs;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p2 = sb + off;
    off += (bytes + 15) & ~size_t(15);
    return p2;
  };
  cs.peak = reinterpret_cast<unsigned long long*>(take(8 * nc));
  cs.sum = reinterpret_cast<double*>(take(8 * nc));
  cs.sx = reinterpret_cast<double*>(take(8 * nc));
  cs.sy = reinterpret_cast<double*>(take(8 * nc));
  cs.count = reinterpret_cast<int*>(take(4 * nc));
  cs.mask_or = reinterpret_cast<unsigned*>(take(4 * nc));
  cs.touched = reinterpret_cast<unsigned*>(take(4 * nc));
  size_t zero_bytes = off;
  cs.first = reinterpret_cast<int*>(take(4 * nc));
  (void)stats_bytes;
  DGPU_CUDA(cudaMemsetAsync(sb, 0, zero_bytes, s));
  DGPU_CUDA(cudaMemsetAsync(cs.first, 0x7f, 4 * nc, s));
  k_comp_reduce<<<kListBlocks, 256, 0, s>>>(w, h, sl, score, mask, cs, c.d_status);
  DGPU_LAUNCH("k_comp_reduce");

  // Output columns: 12 doubles, 4 int32 (peak_x, peak_y, n_pix, psf_chi2_dof), 8 u8.
  const size_t out_bytes = nc * (12 * 8 + 4 * 4 + 8) + 512;
  char* ob = static_cast<char*>(c.slot(kSlotCompOut, out_bytes));
  double* dcol = reinterpret_cast<double*>(ob);
  int* icol = reinterpret_cast<int*>(ob + nc * 12 * 8);
  uint8_t* ucol = reinterpret_cast<uint8_t*>(ob + nc * (12 * 8 + 4 * 4));
  CompOut o;
  o.x = dcol + 0 * nc;
  o.y = dcol + 1 * nc;
  o.peak_snr = dcol + 2 * nc;
  o.flux = dcol + 3 * nc;
  o.expected_n_pix = dcol + 4 * nc;
  o.fwhm_ratio = dcol + 5 * nc;
  o.psf_chi2 = dcol + 6 * nc;
  o.psf_amplitude = dcol + 7 * nc;
  o.psf_amplitude_err = dcol + 8 * nc;
  o.bright_star_dist = dcol + 9 * nc;
  o.peak_x = icol + 0 * nc;
  o.peak_y = icol + 1 * nc;
  o.n_pix = icol + 2 * nc;
  o.psf_chi2_dof = icol + 3 * nc;
  o.fwhm_consistent = ucol + 0 * nc;
  o.mask_flags = ucol + 1 * nc;
  o.is_dipole = ucol + 2 * nc;
  o.quality = ucol + 3 * nc;
  o.shape_consistent = ucol + 4 * nc;
  o.near_bright_star = ucol + 5 * nc;

  FinishParams fp;
  fp.threshold = neg ? p.threshold_sigma_dipole : p.threshold_sigma;
  fp.expected_fwhm = p.expected_fwhm;
  fp.tol_lo = p.fwhm_tolerance_lo;
  fp.tol_hi = p.fwhm_tolerance_hi;
  fp.aperture_radius = p.aperture_radius;
  const bool enrich = ncomp <= std::max(0, p.max_shape_fit);
  fp.do_shape = (enrich && p.fit_psf_shape && psf != nullptr && variance != nullptr && psf_size > 0) ? 1 : 0;
  fp.do_bright = (enrich && bright_x != nullptr && bright_y != nullptr && n_bright > 0) ? 1 : 0;
  fp.shape_tol = p.shape_chi2_tolerance;
  fp.bright_radius = p.bright_star_radius > 0.0 ? p.bright_star_radius : 3.0 * p.expected_fwhm;
  fp.psf_size = psf_size;
  const bool warps = ncomp <= kFinishWarps;
  auto kern = warps ? k_comp_finish<true> : k_comp_finish<false>;
  kern<<<warps ? (ncomp + 3) / 4 : (ncomp + 127) / 128, 128, 0, s>>>(ncomp, w, h, score, diff, mask, variance, psf,
                                                                     bright_x, bright_y, n_bright, cs, fp, o);
  DGPU_LAUNCH("k_comp_finish");
  // Bring the columns back into the context (host).
  std::vector<char> host(out_bytes);
  read_back(c, host.data(), ob, nc * (12 * 8 + 4 * 4 + 8));
  sync_reads(c);
  std::memcpy(c.cat_d.data(), host.data(), nc * 12 * 8);
  std::memcpy(c.cat_i.data(), host.data() + nc * 12 * 8, nc * 4 * 4);
  std::memcpy(c.cat_u8.data(), host.data() + nc * (12 * 8 + 4 * 4), nc * 8);
  return ncomp;
}

}  // namespace dgpu
