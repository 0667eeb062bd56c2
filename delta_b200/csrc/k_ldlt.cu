// Pivoted LDL^T fallback of the batched GLS solver (reference
// src/solve.cpp:177-181 for GCV / fixed lambda, :328-333 for CV folds).
//
// The batched Cholesky (k_solve_cluster) marks a system whose factorisation
// met a non-positive pivot with ok = 0. This kernel then redoes exactly those
// systems the way the reference does when Eigen's LLT fails: Eigen 3.4's
// pivoted LDLT of A = M + lambda P0, theta = A^+ rhs and the effective degrees
// of freedom edf = tr(A^+ M), where A^+ is the LDLT solve with the
// pseudo-inverse of D (1/d where |d| > the smallest normal double, else 0).
// The pivot order is Eigen's: at step k the remaining diagonal entry of
// largest magnitude, read before that step's update (the left-looking variant
// never updates the trailing diagonal early), first on ties. Because that
// order depends on the diagonal alone, it is replayed first and the permuted
// matrix factored without pivoting by a blocked algorithm (the same factors;
// the sums are taken in another order, so they agree to rounding).
//
// It runs after every batched solve, as three launches over chunks of up to
// kLdltChunk systems (a system whose Cholesky succeeded leaves each of them at
// once); a failed system gets a 512-thread CTA for the factorisation and
// theta, then P / 128 CTAs for the trace, with its matrices in a per-system
// global workspace (L2-resident):
//   factor   the pivot order by a sort of the diagonal, then panels of 32
//            columns: the diagonal block by one warp, the rows below by one
//            thread each, the trailing lower triangle minus W L^T on the FP64
//            tensor cores (build_pivoted, ldlt_blocked);
//   theta    forward substitution by one warp (row-oriented), D^+, backward
//            substitution column-oriented by the block, inverse permutation;
//   edf      Z = L^-T D^+ L^-1 (Pi M Pi^T) with one thread per column (no
//            synchronisation between columns), the diagonal summed in a fixed
//            order by the finishing launch.
// A solved system is marked ok = 2, so callers can tell which arithmetic
// produced it. Failed systems are rare for a well-posed fit, but a basis far
// narrower than the pixel scale makes every small-lambda system singular, so
// all of a batch's failures are factored at once.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "dev_common.cuh"
#include "fit_internal.h"

namespace cg = cooperative_groups;

namespace dgpu {

constexpr int kLdltThreads = 512;
constexpr int kLdltMaxP = 1024;
constexpr int kLdltChunk = 32;      // systems per round of the three launches
constexpr int kLdltTraceThreads = 128;

constexpr int kLb = 32;  // panel width of the blocked factorisation

// Per-system workspace: A (P x P, then L and D), Y (P x P), D^+ (P), the trace
// column terms (P), the transposed panels W^T and L^T of the factorisation
// (2 x kLb x P) as doubles; then per system the permutation (P) and a
// factored flag as ints.
__host__ __device__ inline size_t ldlt_sys_doubles(int P) {
  return 2 * static_cast<size_t>(P) * P + 2 * static_cast<size_t>(P) + 2 * static_cast<size_t>(kLb) * P;
}
size_t ldlt_work_bytes(int P, int nsys) {
  return sizeof(double) * ldlt_sys_doubles(P) * nsys + sizeof(int) * (static_cast<size_t>(P) + 1) * nsys;
}

namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

// Block-shared scratch of the factorisation and solves.
struct LdltShared {
  double temp[kLdltMaxP];  // the pivot order's diagonal; later a solve vector
  int piv;                 // -1: the whole diagonal is zero
  int perm[kLdltMaxP];     // position -> original index
};

// The CTAs that share one factorisation: a cluster, or a single CTA.
struct Alone {
  __device__ int rank() const { return 0; }
  __device__ int count() const { return 1; }
  __device__ void sync() const { __syncthreads(); }
};
struct Cluster {
  cg::cluster_group g;
  __device__ int rank() const { return static_cast<int>(g.block_rank()); }
  __device__ int count() const { return static_cast<int>(g.num_blocks()); }
  // Global writes of every CTA visible to the others (which read them past L1).
  __device__ void sync() const {
    __threadfence();
    g.sync();
  }
};

// Eigen's pivot order, from the diagonal alone: its LDLT is left-looking, so
// the trailing diagonal is never updated before its own step and step k's
// pivot (the largest |A_ii| over the positions not yet factored, first on
// ties) depends only on the diagonal of A = M + lambda P0 and the swaps made
// so far. Without equal entries that is the descending order of |A_ii|, one
// bitonic sort; with ties (or NaN) one warp replays the P steps, since the
// swaps then decide which of the equal entries comes first. The permuted
// matrix B = Pi A Pi^T is factored without pivoting. Every CTA of the group
// finds the order for itself and writes its share of B. Returns false when
// the whole diagonal is zero (Eigen then factors nothing).
template <class Group>
__device__ bool build_pivoted(double* B, const double* M, int P, int kk, double lam, const double* pen,
                              LdltShared& S, const Group& grp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* dg = S.temp;
  auto diagonal = [&](int i) { return fma(lam, pen[(i % kk) * kk + (i % kk)], M[static_cast<size_t>(i) * P + i]); };
  int n2 = 2;
  while (n2 < P) n2 <<= 1;
  bool plain = true;  // no NaN and no equal entries
  for (int i = tid; i < n2; i += blockDim.x) {
    const double v = i < P ? fabs(diagonal(i)) : -1.0;
    plain = plain && v == v;
    dg[i] = v;
    S.perm[i] = i;
  }
  if (tid == 0) S.piv = 0;
  __syncthreads();
  for (int size = 2; size <= n2; size <<= 1)
    for (int half = size >> 1; half > 0; half >>= 1) {
      for (int t = tid; t < n2 / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (half - 1)), j = i + half;
        const double vi = dg[i], vj = dg[j];
        if ((i & size) == 0 ? vi < vj : vi > vj) {
          dg[i] = vj;
          dg[j] = vi;
          const int q = S.perm[i];
          S.perm[i] = S.perm[j];
          S.perm[j] = q;
        }
      }
      __syncthreads();
    }
  for (int i = tid; i + 1 < P; i += blockDim.x) plain = plain && dg[i] != dg[i + 1];
  plain = __syncthreads_and(plain);
  if (plain) {
    if (!(dg[0] > 0.0)) return false;  // one unknown, a zero
  } else {
    for (int i = tid; i < P; i += blockDim.x) {
      dg[i] = diagonal(i);
      S.perm[i] = i;
    }
    __syncthreads();
  }
  if (!plain && warp == 0) {
    for (int k = 0; k < P; ++k) {
      double best = -1.0;
      int bi = P;
      for (int i = k + lane; i < P; i += 32) {
        const double v = fabs(dg[i]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
          best = ov;
          bi = oi;
        }
      }
      if (k == 0 && !(best > 0.0)) {
        if (lane == 0) S.piv = -1;
        break;
      }
      if (lane == 0 && bi < P && bi != k) {
        const double t = dg[k];
        dg[k] = dg[bi];
        dg[bi] = t;
        const int q = S.perm[k];
        S.perm[k] = S.perm[bi];
        S.perm[bi] = q;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (S.piv < 0) return false;
  for (int i = grp.rank() + grp.count() * warp; i < P; i += grp.count() * static_cast<int>(blockDim.x >> 5)) {
    const int pi = S.perm[i];
    for (int j = lane; j < P; j += 32) {
      const int pj = S.perm[j];
      double v = M[static_cast<size_t>(pi) * P + pj];
      if (pi / kk == pj / kk) v = fma(lam, pen[(pi % kk) * kk + (pj % kk)], v);
      B[static_cast<size_t>(i) * P + j] = v;
    }
  }
  grp.sync();
  return true;
}

__device__ __forceinline__ void dmma_ldlt(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

constexpr int kLdltRows = 256;  // panel rows a CTA holds at once (dynamic shared memory)
constexpr size_t kLdltDynSmem = sizeof(double) * kLdltRows * (kLb + 1);

// LDL^T of B without pivoting (the lower triangle; L below the diagonal, D on
// it), right-looking over panels of kLb columns by the group's CTAs together:
//   (a) the panel's diagonal block by one warp of every CTA, lane = row with
//       the row in registers, each column's w = d l passed through shared memory;
//   (b) the panel's rows below, split over the CTAs, one thread per row with
//       the row in registers;
//   (c) the trailing lower triangle minus W L^T (W = L D, both panels kept
//       transposed so a column read is contiguous) as m8n8k4 products, 16 x 32
//       per warp over all CTAs.
// Every entry is the FMA chain in ascending column order that one thread would
// form (m8n8k4 rounds like four FMAs in k order). A zero d_k leaves its column
// undivided, as Eigen does. Wt, Lt: kLb x P each. The factorisation is a chain
// of latencies (P / 32 panels of 32 divisions); one CTA with 4 x 4 SIMT blocks
// and the diagonal block's columns in one lane took 2.84 ms at P = 464, a
// cluster of eight 0.60 ms.
template <class Group>
__device__ void ldlt_blocked(double* B, int P, double* Wt, double* Lt, double (*rows)[kLb + 1], const Group& grp) {
  __shared__ double blk[kLb][kLb + 1];  // L of the diagonal block (d on the diagonal)
  __shared__ double wk[kLb][kLb + 1];   // wk[j][k] = d_j l_kj
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), nt = blockDim.x;
  const int rank = grp.rank(), nr = grp.count();
  for (int p0 = 0; p0 < P; p0 += kLb) {
    const int nb = min(kLb, P - p0);
    for (int e = tid; e < kLb * kLb; e += nt) {
      const int r = e / kLb, c = e - r * kLb;
      blk[r][c] = (r < nb && c <= r) ? __ldcg(B + static_cast<size_t>(p0 + r) * P + p0 + c) : 0.0;
    }
    __syncthreads();
    if (warp == 0) {
      double a[kLb];
#pragma unroll
      for (int c = 0; c < kLb; ++c) a[c] = blk[lane][c];
#pragma unroll
      for (int j = 0; j < kLb; ++j) {
        if (j < nb) {
          const double d = __shfl_sync(0xffffffffu, a[j], j);
          const double l = d != 0.0 ? a[j] / d : a[j];
          if (lane > j) {
            wk[j][lane] = d * l;
            a[j] = l;
          }
          __syncwarp();
#pragma unroll
          for (int k = j + 1; k < kLb; ++k)
            if (lane >= k) a[k] = fma(-l, wk[j][k], a[k]);
        }
      }
#pragma unroll
      for (int c = 0; c < kLb; ++c) blk[lane][c] = a[c];
    }
    __syncthreads();
    const int r0 = p0 + nb, T = P - r0;
    const int per = (T + nr - 1) / nr;
    const int i1 = min(P, r0 + (rank + 1) * per);
    for (int ib = r0 + rank * per; ib < i1; ib += kLdltRows) {
      const int n = min(kLdltRows, i1 - ib);
      for (int e = tid; e < n * kLb; e += nt) {
        const int r = e / kLb, c = e - r * kLb;
        rows[r][c] = c < nb ? __ldcg(B + static_cast<size_t>(ib + r) * P + p0 + c) : 0.0;
      }
      __syncthreads();
      if (tid < n) {
        double a[kLb];
#pragma unroll
        for (int c = 0; c < kLb; ++c) a[c] = rows[tid][c];
#pragma unroll
        for (int j = 0; j < kLb; ++j) {
          if (j < nb) {
            const double d = blk[j][j];
            const double l = d != 0.0 ? a[j] / d : a[j];
            a[j] = l;
#pragma unroll
            for (int k = j + 1; k < kLb; ++k) a[k] = fma(-l, wk[j][k], a[k]);  // columns from nb on: unused
            Lt[static_cast<size_t>(j) * P + ib + tid] = l;
            Wt[static_cast<size_t>(j) * P + ib + tid] = l * d;
          }
        }
#pragma unroll
        for (int c = 0; c < kLb; ++c) rows[tid][c] = a[c];
      }
      __syncthreads();
      for (int e = tid; e < n * nb; e += nt) {
        const int r = e / nb, c = e - r * nb;
        B[static_cast<size_t>(ib + r) * P + p0 + c] = rows[r][c];
      }
      __syncthreads();
    }
    grp.sync();  // the panel is complete (and every CTA has read the diagonal block)
    if (rank == 0)
      for (int e = tid; e < nb * nb; e += nt) {
        const int r = e / nb, c = e - r * nb;
        if (c <= r) B[static_cast<size_t>(p0 + r) * P + p0 + c] = blk[r][c];
      }
    if (T > 0) {
      const int n32 = (T + 31) / 32, nu = n32 * (n32 + 1);  // 16 x 32 units of the lower 32 x 32 tiles
      const int q = lane >> 2, kq = lane & 3;
      for (int u = rank + nr * warp; u < nu; u += nr * (nt >> 5)) {
        const int t = u >> 1;
        int ti = static_cast<int>((sqrtf(8.0f * static_cast<float>(t) + 1.0f) - 1.0f) * 0.5f);
        if ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
        if (ti * (ti + 1) / 2 > t) --ti;
        const int tj = t - ti * (ti + 1) / 2;
        const int i0 = r0 + 32 * ti + 16 * (u & 1), j0 = r0 + 32 * tj;
        double acc[2][4][2];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[x][y][0] = acc[x][y][1] = 0.0;
#pragma unroll 2
        for (int k0 = 0; k0 < kLb; k0 += 4) {
          const bool in = k0 + kq < nb;
          const double* wr = Wt + static_cast<size_t>(k0 + kq) * P;
          const double* lr = Lt + static_cast<size_t>(k0 + kq) * P;
          double af[2], bf[4];
#pragma unroll
          for (int x = 0; x < 2; ++x) af[x] = (in && i0 + 8 * x + q < P) ? __ldcg(wr + i0 + 8 * x + q) : 0.0;
#pragma unroll
          for (int y = 0; y < 4; ++y) bf[y] = (in && j0 + 8 * y + q < P) ? __ldcg(lr + j0 + 8 * y + q) : 0.0;
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) dmma_ldlt(acc[x][y], af[x], bf[y]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int ii = i0 + 8 * x + q, jj = j0 + 8 * y + 2 * kq + e;
              if (ii < P && jj <= ii) {
                double* g = B + static_cast<size_t>(ii) * P + jj;
                *g = __ldcg(g) - acc[x][y][e];
              }
            }
      }
    }
    grp.sync();
  }
}

// Pseudo-inverse of D.
__device__ void ldlt_dinv(const double* A, int P, int n_steps, double* dinv) {
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    const double d = n_steps ? __ldcg(A + static_cast<size_t>(i) * P + i) : 0.0;
    dinv[i] = fabs(d) > DBL_MIN ? 1.0 / d : 0.0;
  }
  __syncthreads();
}

struct LdltWork {
  double* d;  // chunk x ldlt_sys_doubles(P)
  int* i;     // chunk x (P + 1): permutation, factored flag
};

// One CTA per system of the chunk [s0, s0 + gridDim.x): factor and theta of a
// failed system; the factored flag tells the next two launches which systems
// to finish.
__global__ void __launch_bounds__(kLdltThreads) k_ldlt_factor(SolveBatch b, int s0, LdltWork wk) {
  extern __shared__ double lrows[][kLb + 1];
  __shared__ LdltShared S;
  const int P = b.P, tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const size_t PP = static_cast<size_t>(P) * P;
  const int s = s0 + static_cast<int>(blockIdx.x);
  double* A = wk.d + blockIdx.x * ldlt_sys_doubles(P);
  double* dinv = A + 2 * PP;
  int* perm = wk.i + blockIdx.x * (static_cast<size_t>(P) + 1);
  int* factored = perm + P;
  if (b.ok[s]) {  // same value for every thread of the block
    if (tid == 0) *factored = 0;
    return;
  }
  const double lam = b.lam[s];
  const double* M = b.M + static_cast<size_t>(b.m_index ? b.m_index[s] : 0) * PP;
  const double* rhs = b.rhs + static_cast<size_t>(b.r_index ? b.r_index[s] : 0) * P;
  double* Wt = A + 2 * PP + 2 * static_cast<size_t>(P);
  const Alone alone;
  const bool any = build_pivoted(A, M, P, b.k, lam, b.pen, S, alone);
  if (any) ldlt_blocked(A, P, Wt, Wt + static_cast<size_t>(kLb) * P, lrows, alone);
  ldlt_dinv(A, P, any ? P : 0, dinv);

  // theta: x = Pi rhs; forward L (unit, row-oriented, one warp); D^+;
  // backward L^T (column t of L^T = row t of L, the block over i < t).
  if (warp == 0) {
    for (int i = 0; i < P; ++i) {
      const double* Ai = A + static_cast<size_t>(i) * P;
      double acc = 0.0;
      for (int j = lane; j < i; j += 32) acc = fma(Ai[j], S.temp[j], acc);
      acc = warp_sum(acc);
      if (lane == 0) S.temp[i] = rhs[S.perm[i]] - acc;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int i = tid; i < P; i += blockDim.x) S.temp[i] *= dinv[i];
  __syncthreads();
  for (int t = P - 1; t > 0; --t) {
    const double zt = S.temp[t];
    const double* At = A + static_cast<size_t>(t) * P;
    for (int i = tid; i < t; i += blockDim.x) S.temp[i] = fma(-At[i], zt, S.temp[i]);
    __syncthreads();
  }
  for (int i = tid; i < P; i += blockDim.x) {
    b.theta[static_cast<size_t>(s) * P + S.perm[i]] = S.temp[i];
    perm[i] = S.perm[i];
  }
  if (tid == 0) *factored = 1;
}

// Y[:, c] <- L^-T D^+ L^-1 Y[:, c] for the thread's column c (Y is P rows of
// stride ldy), the CTA's columns together, by panels of kLb rows. Per panel the
// threads solve its triangular block with their panel values in registers,
// then update the rows still to come with the panel's L read once into shared
// memory (chunks of kTrRows rows): every L value is a broadcast shared load,
// every y value one coalesced load and store. The backward pass stops at the
// panel holding row `stop` (rows above it are left unfinished).
constexpr int kTrRows = 64;

__device__ void panel_solve(const double* A, int P, const double* dinv, double* Y, size_t ldy, int c, bool act,
                            int stop) {
  __shared__ double lp[kLb][kLb + 1];      // the panel's diagonal block
  __shared__ double ls[kTrRows][kLb + 1];  // a chunk of the panel's other rows (forward) / columns (backward)
  const int tid = threadIdx.x, nt = blockDim.x;
  double yp[kLb];
  // Forward: y = L^-1 b (L unit lower).
  for (int p0 = 0; p0 < P; p0 += kLb) {
    const int nb = min(kLb, P - p0);
    __syncthreads();
    for (int e = tid; e < nb * nb; e += nt) {
      const int r = e / nb, q = e - r * nb;
      lp[r][q] = q < r ? A[static_cast<size_t>(p0 + r) * P + p0 + q] : 0.0;
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int k = 0; k < kLb; ++k) {
        if (k < nb) {
          double v = Y[static_cast<size_t>(p0 + k) * ldy + c];
#pragma unroll
          for (int j = 0; j < k; ++j) v = fma(-lp[k][j], yp[j], v);
          yp[k] = v;
          Y[static_cast<size_t>(p0 + k) * ldy + c] = v;
        }
      }
    }
    for (int r0 = p0 + nb; r0 < P; r0 += kTrRows) {
      const int nr = min(kTrRows, P - r0);
      __syncthreads();
      for (int e = tid; e < nr * nb; e += nt) {
        const int r = e / nb, q = e - r * nb;
        ls[r][q] = A[static_cast<size_t>(r0 + r) * P + p0 + q];
      }
      __syncthreads();
      if (act) {
        for (int r = 0; r < nr; ++r) {
          double* yr = Y + static_cast<size_t>(r0 + r) * ldy + c;
          double v = *yr;
#pragma unroll
          for (int k = 0; k < kLb; ++k)
            if (k < nb) v = fma(-ls[r][k], yp[k], v);
          *yr = v;
        }
      }
    }
  }
  // D^+.
  if (act)
    for (int i = 0; i < P; ++i) Y[static_cast<size_t>(i) * ldy + c] *= dinv[i];
  // Backward: x = L^-T y, panels from the last down to the one holding `stop`.
  const int last = ((P - 1) / kLb) * kLb;
  for (int p0 = last; p0 + kLb > stop; p0 -= kLb) {
    const int nb = min(kLb, P - p0);
    __syncthreads();
    for (int e = tid; e < nb * nb; e += nt) {
      const int r = e / nb, q = e - r * nb;
      lp[r][q] = q < r ? A[static_cast<size_t>(p0 + r) * P + p0 + q] : 0.0;
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int kk = kLb - 1; kk >= 0; --kk) {
        if (kk < nb) {
          double v = Y[static_cast<size_t>(p0 + kk) * ldy + c];
#pragma unroll
          for (int t = kk + 1; t < kLb; ++t)
            if (t < nb) v = fma(-lp[t][kk], yp[t], v);
          yp[kk] = v;
          Y[static_cast<size_t>(p0 + kk) * ldy + c] = v;
        }
      }
    }
    // rows r in [stop, p0) above the panel: y_r -= sum_t L[p0 + t][r] x_t
    const int rlo = min(stop, p0);
    for (int r0 = rlo; r0 < p0; r0 += kTrRows) {
      const int nr = min(kTrRows, p0 - r0);
      __syncthreads();
      for (int e = tid; e < nr * nb; e += nt) {
        const int q = e / nr, r = e - q * nr;  // consecutive threads read consecutive columns of row p0 + q
        ls[r][q] = A[static_cast<size_t>(p0 + q) * P + r0 + r];
      }
      __syncthreads();
      if (act) {
        for (int r = 0; r < nr; ++r) {
          double* yr = Y + static_cast<size_t>(r0 + r) * ldy + c;
          double v = *yr;
#pragma unroll
          for (int t = 0; t < kLb; ++t)
            if (t < nb) v = fma(-ls[r][t], yp[t], v);
          *yr = v;
        }
      }
    }
    if (p0 == 0) break;
  }
}

// edf terms Z_cc, Z = L^-T D^+ L^-1 B, B = Pi M Pi^T: thread c solves column c
// (x_c needs x_t, t > c only, so the backward pass stops at the CTA's first
// column). Grid: (chunk systems, ceil(P / kLdltTraceThreads)).
__global__ void __launch_bounds__(kLdltTraceThreads) k_ldlt_trace(SolveBatch b, int s0, LdltWork wk) {
  const int P = b.P;
  const size_t PP = static_cast<size_t>(P) * P;
  const int s = s0 + static_cast<int>(blockIdx.x);
  double* A = wk.d + blockIdx.x * ldlt_sys_doubles(P);
  double* Y = A + PP;
  const double* dinv = A + 2 * PP;
  double* zc = A + 2 * PP + P;
  const int* perm = wk.i + blockIdx.x * (static_cast<size_t>(P) + 1);
  if (!perm[P]) return;  // the same for the whole CTA
  const int c0 = static_cast<int>(blockIdx.y) * kLdltTraceThreads;
  const int c = c0 + static_cast<int>(threadIdx.x);
  const bool act = c < P;
  const double* M = b.M + static_cast<size_t>(b.m_index ? b.m_index[s] : 0) * PP;
  if (act) {
    const int oc = perm[c];
    for (int i = 0; i < P; ++i) Y[static_cast<size_t>(i) * P + c] = M[static_cast<size_t>(perm[i]) * P + oc];
  }
  panel_solve(A, P, dinv, Y, P, c, act, c0);
  if (act) zc[c] = Y[static_cast<size_t>(c) * P + c];
}

// edf = sum_c Z_cc in column order; ok = 2.
__global__ void k_ldlt_finish(SolveBatch b, int s0, LdltWork wk) {
  const int P = b.P;
  const size_t PP = static_cast<size_t>(P) * P;
  const int s = s0 + static_cast<int>(blockIdx.x);
  const int* perm = wk.i + blockIdx.x * (static_cast<size_t>(P) + 1);
  if (threadIdx.x != 0 || !perm[P]) return;
  const double* zc = wk.d + blockIdx.x * ldlt_sys_doubles(P) + 2 * PP + P;
  if (b.want_edf) {
    double e = 0.0;
    for (int c = 0; c < P; ++c) e += zc[c];
    b.edf[s] = e;
  }
  b.ok[s] = 2;
}

// X = A^+ B for A = M + lambda P0: B and X are P x m, row-major, in the
// original order. The same factorisation as the fallback, by one cluster, then
// the columns of B; used where many right-hand sides share one system.
// Workspace: A (P x P), D^+ (P), the factorisation's panels (2 kLb P), the
// permutation (P ints).
constexpr int kSymCluster = 8;

__global__ void __cluster_dims__(kSymCluster, 1, 1) __launch_bounds__(kLdltThreads)
k_sym_factor(int P, int kk, const double* __restrict__ M, double lam, const double* __restrict__ pen, double* A,
             double* dinv, int* __restrict__ perm) {
  extern __shared__ double lrows[][kLb + 1];
  __shared__ LdltShared S;
  const Cluster cl{cg::this_cluster()};
  double* Wt = dinv + P;  // 2 x kLb x P panel workspace
  const bool any = build_pivoted(A, M, P, kk, lam, pen, S, cl);
  if (any) ldlt_blocked(A, P, Wt, Wt + static_cast<size_t>(kLb) * P, lrows, cl);
  if (cl.rank() != 0) return;
  ldlt_dinv(A, P, any ? P : 0, dinv);
  for (int i = threadIdx.x; i < P; i += blockDim.x) perm[i] = S.perm[i];
}

// X[:, c] = A^+ B[:, c] for eight columns per CTA, held in shared memory. Per
// panel of 32 rows: the triangular block by one warp per column (forward) or
// one thread per column (backward, whose sums take the rows in ascending
// order, so each unknown waits for the one before it), then the other rows
// minus L times the panel's values as m8n8k4 products, eight rows per warp.
// Each entry is the FMA chain in ascending order that a thread per column
// would form; that version's 3 CTAs at 378 columns took 3.3 ms, this one's 48
// take 0.18 ms.
constexpr int kScCols = 8;
constexpr int kScLd = 12;  // conflict-free B fragments
constexpr int kScThreads = 512;

__global__ void __launch_bounds__(kScThreads) k_sym_solve_cols(int P, const double* __restrict__ A,
                                                               const double* __restrict__ dinv,
                                                               const int* __restrict__ perm,
                                                               const double* __restrict__ B, int m,
                                                               double* __restrict__ X) {
  extern __shared__ __align__(16) double Y[];  // P x kScLd
  __shared__ double lp[kLb][kLb + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, kq = lane & 3;
  constexpr int kWarps = kScThreads / 32;
  const int c0 = static_cast<int>(blockIdx.x) * kScCols;
  for (int e = tid; e < P * kScCols; e += kScThreads) {
    const int i = e / kScCols, c = e - i * kScCols;
    Y[i * kScLd + c] = c0 + c < m ? B[static_cast<size_t>(perm[i]) * m + c0 + c] : 0.0;
  }
  auto load_block = [&](int p0, int nb) {
    for (int e = tid; e < kLb * kLb; e += kScThreads) {
      const int r = e / kLb, c = e - r * kLb;
      lp[r][c] = (r < nb && c < r) ? A[static_cast<size_t>(p0 + r) * P + p0 + c] : 0.0;
    }
    __syncthreads();
  };
  // Rows [r0, r0 + 8): Y -= L (8 x 32) times the panel's rows of Y; l(row, t) is L's entry.
  auto update = [&](int r0, int rend, int p0, int nb, auto l) {
    double af[8], acc[2];
    const int r = r0 + q;
#pragma unroll
    for (int s = 0; s < 8; ++s) af[s] = (r < rend && 4 * s + kq < nb) ? -l(r, 4 * s + kq) : 0.0;
    double2 y = r < rend ? *reinterpret_cast<const double2*>(Y + r * kScLd + 2 * kq) : make_double2(0.0, 0.0);
    acc[0] = y.x;
    acc[1] = y.y;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int t = 4 * s + kq;
      dmma_ldlt(acc, af[s], t < nb ? Y[(p0 + t) * kScLd + q] : 0.0);
    }
    if (r < rend) *reinterpret_cast<double2*>(Y + r * kScLd + 2 * kq) = make_double2(acc[0], acc[1]);
  };
  // Forward: y = L^-1 b (L unit lower).
  for (int p0 = 0; p0 < P; p0 += kLb) {
    const int nb = min(kLb, P - p0);
    load_block(p0, nb);
    if (warp < kScCols) {
      double v = lane < nb ? Y[(p0 + lane) * kScLd + warp] : 0.0;
#pragma unroll 8
      for (int j = 0; j < nb; ++j) {
        const double yj = __shfl_sync(0xffffffffu, v, j);
        if (lane > j) v = fma(-lp[lane][j], yj, v);
      }
      if (lane < nb) Y[(p0 + lane) * kScLd + warp] = v;
    }
    __syncthreads();
    for (int r0 = p0 + nb + 8 * warp; r0 < P; r0 += 8 * kWarps)
      update(r0, P, p0, nb, [&](int r, int t) { return A[static_cast<size_t>(r) * P + p0 + t]; });
    __syncthreads();
  }
  // D^+.
  for (int e = tid; e < P * kScCols; e += kScThreads) {
    const int i = e / kScCols;
    Y[i * kScLd + e - i * kScCols] *= dinv[i];
  }
  // Backward: x = L^-T y.
  for (int p0 = ((P - 1) / kLb) * kLb; p0 >= 0; p0 -= kLb) {
    const int nb = min(kLb, P - p0);
    load_block(p0, nb);
    if (tid < kScCols) {
      double yp[kLb];
#pragma unroll
      for (int kk = kLb - 1; kk >= 0; --kk) {
        if (kk < nb) {
          double v = Y[(p0 + kk) * kScLd + tid];
#pragma unroll
          for (int t = kk + 1; t < kLb; ++t)
            if (t < nb) v = fma(-lp[t][kk], yp[t], v);
          yp[kk] = v;
          Y[(p0 + kk) * kScLd + tid] = v;
        }
      }
    }
    __syncthreads();
    for (int r0 = 8 * warp; r0 < p0; r0 += 8 * kWarps)
      update(r0, p0, p0, nb, [&](int r, int t) { return A[static_cast<size_t>(p0 + t) * P + r]; });
    __syncthreads();
  }
  for (int e = tid; e < P * kScCols; e += kScThreads) {
    const int i = e / kScCols, c = e - i * kScCols;
    if (c0 + c < m) X[static_cast<size_t>(perm[i]) * m + c0 + c] = Y[i * kScLd + c];
  }
}

void launch_sym_solve_many(Context& c, int P, int k, const double* M, double lam, const double* pen, const double* B,
                           int m, double* X) {
  if (P > kLdltMaxP) fail(DGPU_ERR_INVALID, "solve: at most 1024 unknowns are supported");
  const size_t PP = static_cast<size_t>(P) * P;
  char* work = static_cast<char*>(
      c.slot(kSlotGrad6, sizeof(double) * (PP + P + 2 * static_cast<size_t>(kLb) * P) + sizeof(int) * P + 16));
  double* A = reinterpret_cast<double*>(work);
  double* dinv = A + PP;
  int* perm = reinterpret_cast<int*>(dinv + P + 2 * static_cast<size_t>(kLb) * P);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_sym_factor), kLdltDynSmem);
  k_sym_factor<<<kSymCluster, kLdltThreads, kLdltDynSmem, c.stream>>>(P, k, M, lam, pen, A, dinv, perm);
  DGPU_LAUNCH("k_sym_factor");
  if (m <= 0) return;
  const size_t smem = sizeof(double) * kScLd * static_cast<size_t>(P);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_sym_solve_cols), smem);
  k_sym_solve_cols<<<(m + kScCols - 1) / kScCols, kScThreads, smem, c.stream>>>(P, A, dinv, perm, B, m, X);
  DGPU_LAUNCH("k_sym_solve_cols");
}

void launch_ldlt_fallback(Context& c, const SolveBatch& b) {
  if (b.nsys <= 0) return;
  if (b.P > kLdltMaxP) fail(DGPU_ERR_INVALID, "solve: the LDLT fallback supports at most 1024 unknowns");
  const int chunk = std::min(b.nsys, kLdltChunk);
  char* work = static_cast<char*>(c.slot(kSlotLdlt, ldlt_work_bytes(b.P, chunk)));
  LdltWork wk;
  wk.d = reinterpret_cast<double*>(work);
  wk.i = reinterpret_cast<int*>(work + sizeof(double) * ldlt_sys_doubles(b.P) * chunk);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_ldlt_factor), kLdltDynSmem);
  for (int s0 = 0; s0 < b.nsys; s0 += chunk) {
    const int m = std::min(chunk, b.nsys - s0);
    k_ldlt_factor<<<m, kLdltThreads, kLdltDynSmem, c.stream>>>(b, s0, wk);
    DGPU_LAUNCH("k_ldlt_factor");
    if (b.want_edf) {
      k_ldlt_trace<<<dim3(m, (b.P + kLdltTraceThreads - 1) / kLdltTraceThreads), kLdltTraceThreads, 0, c.stream>>>(
          b, s0, wk);
      DGPU_LAUNCH("k_ldlt_trace");
    }
    k_ldlt_finish<<<m, 32, 0, c.stream>>>(b, s0, wk);
    DGPU_LAUNCH("k_ldlt_finish");
  }
}

}  // namespace dgpu
