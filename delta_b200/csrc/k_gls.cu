// GCV / CV evaluation kernels on top of the batched solver:
//   * rss and GCV per system (src/solve.cpp:183-191):
//       rss = max(ywy - 2 theta.rhs + theta^T M theta, 0),
//       gcv = n rss / (n - edf)^2 (inf when n <= edf or the factorisation failed);
//   * CV held-out error per (lambda, fold) (src/solve.cpp:334-335);
//   * fold training systems M - M_g, rhs - rhs_g (src/solve.cpp:300-305);
//   * per-stamp moments and the Kronecker fold assembly of the stamped CV
//     solve (src/solve.cpp:584-629).
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "fit_internal.h"
#include "gls_internal.h"

namespace dgpu {

__device__ double block_sum(double v, double* red) {
  red[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < static_cast<unsigned>(o)) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  const double r = red[0];
  __syncthreads();
  return r;
}

// theta^T Mq theta - 2 theta . rq + yq for system s (M/r/y chosen by index).
// With an anchor theta0 (one per r index) the vector is theta - theta0: given
// rq = X^T W e0 and yq = e0^T W e0 for the residual e0 = t - X theta0, that is
// the rss of theta expanded around theta0, whose quadratic term is small near
// the anchor.
// Grid (row blocks of kQRows, systems): each CTA forms the partial sums of its
// rows (one warp per row of M, coalesced); k_quad_finish adds the row blocks
// of each system in a fixed order.
constexpr int kQRows = 32;

__global__ void __launch_bounds__(256)
k_quad_err(int P, const double* __restrict__ theta, const double* __restrict__ M, const int* __restrict__ m_index,
           const double* __restrict__ r, const int* __restrict__ r_index, const double* __restrict__ anchor,
           double* __restrict__ part) {
  __shared__ double red[256];
  __shared__ double th[1024];
  const int b = blockIdx.x, s = blockIdx.y, nb = gridDim.x;
  const double* Mq = M + (m_index ? static_cast<size_t>(m_index[s]) * P * P : 0);
  const double* rq = r + (r_index ? static_cast<size_t>(r_index[s]) * P : 0);
  const double* aq = anchor ? anchor + (r_index ? static_cast<size_t>(r_index[s]) * P : 0) : nullptr;
  for (int p = threadIdx.x; p < P; p += blockDim.x)
    th[p] = theta[static_cast<size_t>(s) * P + p] - (aq ? aq[p] : 0.0);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int p0 = b * kQRows, p1 = min(P, p0 + kQRows);
  double quad = 0.0, lin = 0.0;
  for (int p = p0 + warp; p < p1; p += nw) {
    const double* row = Mq + static_cast<size_t>(p) * P;
    double a = 0.0;
    for (int q = lane; q < P; q += 32) a = fma(row[q], th[q], a);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) quad = fma(th[p], a, quad);
  }
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) lin = fma(th[p], rq[p], lin);
  const double Q = block_sum(quad, red);
  const double L = block_sum(lin, red);
  if (threadIdx.x == 0) {
    part[(static_cast<size_t>(s) * nb + b) * 2] = Q;
    part[(static_cast<size_t>(s) * nb + b) * 2 + 1] = L;
  }
}

__global__ void k_quad_finish(int nsys, int nb, const double* __restrict__ part, const double* __restrict__ y,
                              const int* __restrict__ r_index, double* __restrict__ out) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsys; s += gridDim.x * blockDim.x) {
    double Q = 0.0, L = 0.0;
    for (int b = 0; b < nb; ++b) {
      Q += part[(static_cast<size_t>(s) * nb + b) * 2];
      L += part[(static_cast<size_t>(s) * nb + b) * 2 + 1];
    }
    out[s] = y[r_index ? r_index[s] : 0] - 2.0 * L + Q;
  }
}

// theta0 = theta of the first system with the smallest curve value (NaN never
// wins; all-NaN picks system 0), the host's argmin rule.
__global__ void k_argmin_copy(int nsys, const double* __restrict__ curve, const double* __restrict__ theta, int P,
                              double* __restrict__ theta0) {
  __shared__ int s_best;
  if (threadIdx.x == 0) {
    int b = 0;
    double bg = __longlong_as_double(0x7ff0000000000000ll);
    for (int i = 0; i < nsys; ++i)
      if (curve[i] < bg) {
        bg = curve[i];
        b = i;
      }
    s_best = b;
  }
  __syncthreads();
  const double* src = theta + static_cast<size_t>(s_best) * P;
  for (int p = threadIdx.x; p < P; p += blockDim.x) theta0[p] = src[p];
}

void launch_argmin_copy(cudaStream_t st, int nsys, const double* curve, const double* theta, int P,
                        double* theta0) {
  k_argmin_copy<<<1, 256, 0, st>>>(nsys, curve, theta, P, theta0);
  DGPU_LAUNCH("k_argmin_copy");
}

void launch_quad_err(Context& c, int nsys, int P, const double* theta, const double* M, const int* m_index,
                     const double* r, const int* r_index, const double* y, double* out, const double* anchor) {
  if (nsys == 0) return;
  const int nb = (P + kQRows - 1) / kQRows;
  double* part = static_cast<double*>(c.slot(kSlotGlsPart, sizeof(double) * 2 * static_cast<size_t>(nb) * nsys));
  k_quad_err<<<dim3(nb, nsys), 256, 0, c.stream>>>(P, theta, M, m_index, r, r_index, anchor, part);
  DGPU_LAUNCH("k_quad_err");
  k_quad_finish<<<(nsys + 127) / 128, 128, 0, c.stream>>>(nsys, nb, part, y, r_index, out);
  DGPU_LAUNCH("k_quad_finish");
}

__global__ void k_gcv_finish(int nsys, const double* __restrict__ raw, const double* __restrict__ edf,
                             const int* __restrict__ ok, const long long* __restrict__ n, double* __restrict__ rss,
                             double* __restrict__ gcv) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  double r = raw[s];
  if (r < 0.0) r = 0.0;
  rss[s] = r;
  const double nn = static_cast<double>(*n);
  const double denom = nn - edf[s];
  gcv[s] = (ok[s] && denom > 0.0) ? nn * r / (denom * denom) : __longlong_as_double(0x7ff0000000000000ll);
}

void launch_gcv_finish(cudaStream_t st, int nsys, const double* raw, const double* edf, const int* ok,
                       const long long* n, double* rss, double* gcv) {
  k_gcv_finish<<<(nsys + 127) / 128, 128, 0, st>>>(nsys, raw, edf, ok, n, rss, gcv);
  DGPU_LAUNCH("k_gcv_finish");
}

// out[g] = all - part[g] for g < groups (matrices or vectors of length len).
__global__ void k_sub_parts(int groups, size_t len, const double* __restrict__ all, const double* __restrict__ part,
                            double* __restrict__ out) {
  const size_t total = static_cast<size_t>(groups) * len;
  for (size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[e] = all[e % len] - part[e];
}

__global__ void k_sum_parts(int groups, size_t len, const double* __restrict__ part, double* __restrict__ all) {
  for (size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < len;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    double s = 0.0;
    for (int g = 0; g < groups; ++g) s += part[static_cast<size_t>(g) * len + e];
    all[e] = s;
  }
}

void launch_fold_train(cudaStream_t st, int groups, size_t len, const double* part, double* all, double* train) {
  const int blocks = static_cast<int>(std::min<size_t>((len + 255) / 256, 148 * 8));
  k_sum_parts<<<std::max(blocks, 1), 256, 0, st>>>(groups, len, part, all);
  DGPU_LAUNCH("k_sum_parts");
  const int b2 = static_cast<int>(std::min<size_t>((groups * len + 255) / 256, 148 * 8));
  k_sub_parts<<<std::max(b2, 1), 256, 0, st>>>(groups, len, all, part, train);
  DGPU_LAUNCH("k_sub_parts");
}

// Per-stamp moments over the stamp's active rows: A_s = sum w b b^T (nf x nf,
// full), r_s = sum w t b, ds2_s = sum w t^2, pixel-centroid sums. A CTA per stamp:
// with t appended to the row, [b, t], all three are one product (w [b, t])^T
// [b, t] with the rows as the inner dimension, on the FP64 tensor cores, each
// entry the FMA chain over the rows in order. Rows arrive by cp.async, kSmRows at a
// time. Bound by reading the rows (230 bytes each; 200 stamps of 961 rows, 29
// fields: 44 MB, 7 us at 6.5 TB/s) and one chain of DMMAs per entry; a thread per entry walking the rows took
// 2.1 ms, this 0.09 ms.
constexpr int kSmRows = 64;
constexpr int kSmThreads = 512;

__host__ __device__ inline int sm_ld(int nf) { return ((nf + 1 + 7) / 8 * 8 + 11) / 16 * 16 + 4; }  // >= nf + 1 rounded to 8, = 4 mod 16
size_t stamp_moments_smem(int nf) { return sizeof(double) * kSmRows * (3 * static_cast<size_t>(sm_ld(nf)) + 2); }

__device__ __forceinline__ void dmma_gls(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(kSmThreads)
k_stamp_moments(int nc, int SS, FitRows R, const uint8_t* __restrict__ accepted, double* __restrict__ As,
                double* __restrict__ rs, double* __restrict__ ds2, double* __restrict__ cen) {
  extern __shared__ __align__(16) double smm[];
  const int s = blockIdx.x, nf = nc + 1, ld = sm_ld(nf), nt = (nf + 1 + 7) / 8;  // tiles of 8 per side
  double* rows = smm;                          // 2 x kSmRows x ld: b (background 1), t, zeros
  double* wrow = rows + 2 * kSmRows * ld;      // kSmRows x ld: w [b, t]
  double* wv = wrow + kSmRows * ld;            // 2 x kSmRows: w
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, kq = lane & 3;
  constexpr int kWarps = kSmThreads / 32;
  const size_t base = static_cast<size_t>(s) * SS;
  const bool on = accepted[s] != 0;
  const int n = on ? SS : 0;
  auto active = [&](int i) { return i < n && R.valid[base + i]; };
  // Inactive rows stay out of shared memory (zeros there) and out of every sum.
  auto stage = [&](int i0, int buf) {
    for (int rr = warp; rr < kSmRows; rr += kWarps) {
      double* o = rows + (buf * kSmRows + rr) * ld;
      const size_t row = base + i0 + rr;
      if (active(i0 + rr)) {
        for (int c = lane; c < nc; c += 32)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(o + c))),
                       "l"(R.bn + row * nc + c) : "memory");
        if (lane == 0) {
          o[nc] = 1.0;
          o[nf] = R.t[row];
          wv[buf * kSmRows + rr] = R.w[row];
        }
      } else {
        for (int c = lane; c < ld; c += 32) o[c] = 0.0;
        if (lane == 0) wv[buf * kSmRows + rr] = 0.0;
      }
      for (int c = nf + 1 + lane; c < ld; c += 32) o[c] = 0.0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // This warp's output tiles: warp, warp + kWarps, ... of nt x nt, kMost at a time.
  constexpr int kMost = 4;
  double cx = 0.0, cy = 0.0, cn = 0.0;
  for (int t0 = 0; t0 < nt * nt; t0 += kMost * kWarps) {
    double acc[kMost][2];
#pragma unroll
    for (int u = 0; u < kMost; ++u) acc[u][0] = acc[u][1] = 0.0;
    __syncthreads();
    if (n > 0) stage(0, 0);
    int buf = 0;
    for (int i0 = 0; i0 < n; i0 += kSmRows) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // this chunk is in place, the previous one is read
      const double* cur = rows + buf * kSmRows * ld;
      const double* cw = wv + buf * kSmRows;
      for (int e = tid; e < kSmRows * 8 * nt; e += kSmThreads) {
        const int rr = e / (8 * nt), c = e - rr * 8 * nt;
        wrow[rr * ld + c] = cw[rr] * cur[rr * ld + c];
      }
      if (t0 == 0 && tid < kSmRows && active(i0 + tid)) {
        cx += static_cast<double>(R.px[base + i0 + tid]);
        cy += static_cast<double>(R.py[base + i0 + tid]);
        cn += 1.0;
      }
      buf ^= 1;
      if (i0 + kSmRows < n) stage(i0 + kSmRows, buf);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kMost; ++u) {
        const int t = t0 + u * kWarps + warp;
        if (t >= nt * nt) break;
        const double* A = wrow + kq * ld + 8 * (t / nt) + q;
        const double* B = cur + kq * ld + 8 * (t % nt) + q;
#pragma unroll
        for (int k0 = 0; k0 < kSmRows; k0 += 4) dmma_gls(acc[u], A[k0 * ld], B[k0 * ld]);
      }
    }
#pragma unroll
    for (int u = 0; u < kMost; ++u) {
      const int t = t0 + u * kWarps + warp;
      if (t >= nt * nt) break;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int a = 8 * (t / nt) + q, b = 8 * (t % nt) + 2 * kq + e;
        if (a < nf && b < nf)
          As[(static_cast<size_t>(s) * nf + a) * nf + b] = acc[u][e];
        else if (a == nf && b < nf)
          rs[static_cast<size_t>(s) * nf + b] = acc[u][e];
        else if (a == nf && b == nf)
          ds2[s] = acc[u][e];
      }
    }
  }
  // Centroid sums: whole numbers, exact in any order.
  __shared__ double red[3][2];
  if (warp < 2) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cx += __shfl_xor_sync(0xffffffffu, cx, o);
      cy += __shfl_xor_sync(0xffffffffu, cy, o);
      cn += __shfl_xor_sync(0xffffffffu, cn, o);
    }
    if (lane == 0) {
      red[0][warp] = cx;
      red[1][warp] = cy;
      red[2][warp] = cn;
    }
  }
  __syncthreads();
  if (tid < 3) cen[static_cast<size_t>(s) * 3 + tid] = red[tid][0] + red[tid][1];
}

void launch_stamp_moments(cudaStream_t st, int n_stamps, int nc, int SS, const FitRows& R, const uint8_t* accepted,
                          double* As, double* rs, double* ds2, double* cen) {
  if (n_stamps == 0) return;
  const size_t smem = stamp_moments_smem(nc + 1);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_stamp_moments), smem);
  k_stamp_moments<<<n_stamps, kSmThreads, smem, st>>>(nc, SS, R, accepted, As, rs, ds2, cen);
  DGPU_LAUNCH("k_stamp_moments");
}

// Fold assembly M_g = sum_{s in g} A_s (x) d_s d_s^T, rf_g(c-block) = sum r_s(c) d_s,
// ysq_g = sum ds2_s (src/solve.cpp:605-629), the stamps of a fold in order:
// list[offs[g] .. offs[g + 1]). A CTA takes kSaPairs field pairs (c, c') of one
// fold, a thread one design pair (m, m') of them at a time, so a product d_m d_m'
// serves kSaPairs sums; the last CTA of a fold forms rf and ysq. (A thread per
// entry of M scanning every stamp took 0.22 ms at 5 folds of 40 stamps, P =
// 725; this 0.03 ms.)
constexpr int kSaPairs = 8;
constexpr int kSaStamps = 64;  // stamps staged at a time

__global__ void __launch_bounds__(256)
k_stamped_assemble(int nf, int k, const int* __restrict__ list, const int* __restrict__ offs,
                   const double* __restrict__ As, const double* __restrict__ rs, const double* __restrict__ ds2,
                   const double* __restrict__ dsd, double* __restrict__ Mg, double* __restrict__ rg,
                   double* __restrict__ yg) {
  extern __shared__ __align__(16) double sa[];
  double* sA = sa;                          // kSaStamps x kSaPairs
  double* sd = sA + kSaStamps * kSaPairs;   // kSaStamps x k
  const int g = blockIdx.y, P = nf * k, tid = threadIdx.x;
  const int b0 = offs[g], b1 = offs[g + 1];
  if (blockIdx.x == gridDim.x - 1) {
    for (int p = tid; p <= P; p += 256) {
      const int c = p / k, m = p - c * k;
      double acc = 0.0;
      for (int i = b0; i < b1; ++i) {
        const int s = list[i];
        if (p < P)
          acc += rs[static_cast<size_t>(s) * nf + c] * dsd[static_cast<size_t>(s) * k + m];
        else
          acc += ds2[s];
      }
      if (p < P)
        rg[static_cast<size_t>(g) * P + p] = acc;
      else
        yg[g] = acc;
    }
    return;
  }
  const int e0 = blockIdx.x * kSaPairs, ne = min(kSaPairs, nf * nf - e0);
  for (int mm0 = 0; mm0 < k * k; mm0 += 256) {
    const int mm = mm0 + tid, m = mm / k, m2 = mm - m * k;
    const bool in = mm < k * k;
    double acc[kSaPairs];
#pragma unroll
    for (int e = 0; e < kSaPairs; ++e) acc[e] = 0.0;
    for (int i0 = b0; i0 < b1; i0 += kSaStamps) {
      const int n = min(kSaStamps, b1 - i0);
      __syncthreads();
      for (int t = tid; t < n * kSaPairs; t += 256) {
        const int i = t / kSaPairs, e = t - i * kSaPairs;
        sA[t] = e < ne ? As[static_cast<size_t>(list[i0 + i]) * nf * nf + e0 + e] : 0.0;
      }
      for (int t = tid; t < n * k; t += 256) {
        const int i = t / k;
        sd[t] = dsd[static_cast<size_t>(list[i0 + i]) * k + (t - i * k)];
      }
      __syncthreads();
      if (in)
        for (int i = 0; i < n; ++i) {
          const double dd = sd[i * k + m] * sd[i * k + m2];
#pragma unroll
          for (int e = 0; e < kSaPairs; ++e) acc[e] = fma(sA[i * kSaPairs + e], dd, acc[e]);
        }
    }
    if (in)
      for (int e = 0; e < ne; ++e) {
        const int c = (e0 + e) / nf, c2 = (e0 + e) - c * nf;
        double v = 0.0;
#pragma unroll
        for (int x = 0; x < kSaPairs; ++x) v = x == e ? acc[x] : v;
        Mg[static_cast<size_t>(g) * P * P + static_cast<size_t>(c * k + m) * P + c2 * k + m2] = v;
      }
  }
}

void launch_stamped_assemble(cudaStream_t st, int groups, int nf, int k, const int* list, const int* offs,
                             const double* As, const double* rs, const double* ds2, const double* dsd, double* Mg,
                             double* rg, double* yg) {
  const size_t smem = sizeof(double) * kSaStamps * (kSaPairs + static_cast<size_t>(k));
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_stamped_assemble), smem);
  k_stamped_assemble<<<dim3((nf * nf + kSaPairs - 1) / kSaPairs + 1, groups), 256, smem, st>>>(nf, k, list, offs, As, rs,
                                                                                      ds2, dsd, Mg, rg, yg);
  DGPU_LAUNCH("k_stamped_assemble");
}

// theta += delta (refinement).
__global__ void k_axpy(int n, const double* __restrict__ d, double* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += d[i];
}

// r = r - lam * P0 theta  (P0 = blockdiag pen), for the refinement residual.
__global__ void k_sub_penalty(int P, int k, const double* __restrict__ pen, double lam, const double* __restrict__ th,
                              double* __restrict__ r) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  const int b = p / k, m = p % k;
  double a = 0.0;
  for (int q = 0; q < k; ++q) a = fma(pen[m * k + q], th[b * k + q], a);
  r[p] -= lam * a;
}

void launch_refine_update(cudaStream_t st, int P, int k, const double* pen, double lam, const double* theta,
                          double* r) {
  k_sub_penalty<<<(P + 255) / 256, 256, 0, st>>>(P, k, pen, lam, theta, r);
  DGPU_LAUNCH("k_sub_penalty");
}

void launch_axpy(cudaStream_t st, int n, const double* d, double* x) {
  k_axpy<<<(n + 255) / 256, 256, 0, st>>>(n, d, x);
  DGPU_LAUNCH("k_axpy");
}

}  // namespace dgpu
