// Batched penalised-GLS solver on the device (reference src/solve.cpp:147-193,
// 227-262): for every system s of a batch (the lambda grid, or the lambda x
// fold grid of a CV search)
//   A_s = M_s + lambda_s P0,  A_s = L L^T (FP64 Cholesky),
//   theta_s = L^-T L^-1 rhs_s,  edf_s = P - lambda_s ||L^-1 F||_F^2
// (the reference's exact trace identity, F F^T = P0).
//
// One thread-block cluster per system (systems never wait on each other), of up to
// 16 CTAs. The matrix lives in global memory (L2-resident) as 32 x 32 FP64 tiles and
// is factored by a left-looking blocked Cholesky: column j's tiles
//   C_ij = A_ij - sum_{p<j} L_ip L_jp^T
// are summed in registers and stored once, as L_ij = C_ij Dinv_j^T (Dinv_j =
// L_jj^-1). Below A the rows E = [rhs^T; F^T] are appended and take the same steps,
// which turn them into E L^-T = [(L^-1 rhs)^T; (L^-1 F)^T], so y = L^-1 rhs and the
// trace come out of the factorisation with no inverse of L. E's F rows are zero left
// of their field block, and tiles left of that never enter the computation.
//   Rank 0 sums and factors the diagonal tiles and takes no rows; the other ranks
// deal a column's row tiles among them, up to four at a time against the same L_jp
// tile, and sum column j + 1 ahead while column j is being finished. The chain that
// bounds a factorisation is: Dinv_j to rank 1, L_{j+1,j} back to rank 0, the
// diagonal tile's last product, its 32 pivots. These two transfers go straight into
// the other CTA's shared memory; one cluster barrier per column says that the rest
// of it is stored.
//   What bounds it: with few systems that chain (about 15000 cycles a column at 725
// unknowns), with many the FP64 tensor cores. A right-looking version read and wrote
// every trailing tile once per column, 36 KB of L2 traffic for a product of 0.27 us,
// and waited for two cluster barriers and 18500 cycles of factoring per column: 65
// systems of 725 unknowns without the F rows 1340 -> 865 us, 10 systems 498 -> 390,
// 5 systems 497 -> 340, one with the F rows 762 -> 420; 25 of 475 with them 360 ->
// 305, 25 of 150 82 -> 64.
// The workspace is tile-major (each tile one contiguous block with the
// shared-memory row stride), so tile operands are staged by single bulk async
// copies completing on mbarriers, several columns ahead; products run on the FP64
// tensor cores (mma.sync m8n8k4). A is never assembled: M, converted to tiles once
// per distinct matrix, is read at a tile's column and the penalty added there; E is
// generated there. theta = L^-T y by back substitution on rank 0. The trace is
// reduced per rank in a fixed order and summed in rank order (deterministic). A
// non-positive pivot marks the system failed (ok = 0); k_ldlt.cu then redoes it by
// pivoted LDL^T, as the reference falls back from LLT to LDLT.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "dev_common.cuh"
#include "fit_internal.h"

namespace cg = cooperative_groups;

namespace dgpu {

constexpr int kT = 32;    // tile side
constexpr int kLd = 36;   // shared tile row stride (doubles): 16-byte rows, conflict-free fragments
constexpr int kTS = kT * kLd;
constexpr int kSolveThreads = 256;
constexpr int kMaxTiles = 40;  // tile rows of E (and columns of A) per system

// Workspace, tile-major: every 32 x 32 tile is one contiguous kTS block with
// the shared-memory row stride kLd, so a tile moves with one bulk copy. Per
// system: the lower tiles of A (row-major triangle), the ne x nb tiles of E,
// the nb tiles of Dinv; then the lower tiles of each distinct M (identity
// padding outside P x P).
int solve_pp(int P) { return (P + kT - 1) / kT * kT; }
int solve_ep(int nf, int r) { return (nf * r + 1 + kT - 1) / kT * kT; }
size_t solve_sys_doubles(int P, int nf, int r) {
  const size_t nb = solve_pp(P) / kT, ne = solve_ep(nf, r) / kT;
  return (nb * (nb + 1) / 2 + ne * nb + nb) * kTS;
}
size_t solve_m_doubles(int P) {
  const size_t nb = solve_pp(P) / kT;
  return nb * (nb + 1) / 2 * kTS;
}
size_t solve_work_doubles(int P, int nf, int r, int nsys, int nm) {
  return static_cast<size_t>(nsys) * solve_sys_doubles(P, nf, r) + static_cast<size_t>(std::max(nm, 1)) * solve_m_doubles(P);
}
__host__ __device__ __forceinline__ int tri_index(int ti, int tj) { return ti * (ti + 1) / 2 + tj; }

constexpr int kGroup = 4;         // row tiles a CTA updates together
constexpr int kStages = 8;        // operand stages in flight, at most
constexpr int kRingSmall = 10;    // shared tiles for operands in flight, two CTAs on an SM
constexpr int kRingLarge = 22;    // and one

struct SolveSmem {
  double d[kTS];            // Dinv_j; on the factoring rank the diagonal tile
  double nx[kTS];           // factoring rank: L_{j,j-1}
  double red[kSolveThreads];
  // Mbarriers: the operand stages, the arrival of d and nx, the factoring rank's L_{j,j-2}.
  uint64_t full[kStages], empty[kStages], dbar, nbar, pbar;
  alignas(16) double ring[1][kTS];  // operand stages; panel operands; the factoring rank's other tiles
};
// The factoring rank's use of the ring: factor_tile's three tiles, Dinv_j on its
// way to the others, the next diagonal tile's sum, then L_{j,j-2} and the stages.
enum { kRingDinv = 3, kRingDiag = 4, kRingPrev = 5, kRingStages = 6 };
size_t solve_smem(int ring) { return sizeof(SolveSmem) + (ring - 1) * sizeof(double) * kTS; }

constexpr long long kSolveSpin = 1ll << 22;  // bounded mbarrier wait (iterations)

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// 1-D bulk async copy global -> this CTA's shared memory completing on `bar`
// (no multicast); dst, src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(saddr(dst)), "l"(src), "r"(bytes), "r"(saddr(bar))
               : "memory");
}
// The same from this CTA's shared memory to the same place in rank r's, completing
// on rank r's `bar`.
__device__ __forceinline__ void bulk_s2rank(void* dst, const void* src, uint32_t bytes, uint64_t* bar, int r) {
  uint32_t rd, rb;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rd) : "r"(saddr(dst)), "r"(r));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(saddr(bar)), "r"(r));
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(rd), "r"(saddr(src)), "r"(bytes), "r"(rb)
               : "memory");
}
// Generic-proxy accesses of this CTA (ordered by a preceding barrier) before
// the async-proxy writes the issuing thread starts next.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase of `bar` with the given parity; false on expiry.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  const uint32_t a = saddr(bar);
  for (long long it = 0; it < kSolveSpin; ++it) {
    uint32_t done = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// The same where another CTA of the cluster arrives.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, unsigned parity) {
  const uint32_t a = saddr(bar);
  for (long long it = 0; it < kSolveSpin; ++it) {
    uint32_t done = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

constexpr uint32_t kTileBytes = kTS * sizeof(double);
constexpr size_t kTSz = kTS;

// The warp's index as a value the compiler knows to be uniform. Behind a branch on
// threadIdx.x / 32 it must assume a diverged warp, and each shuffle or warp barrier
// there then costs some 200 cycles (16 pivots of a tile: 14000 cycles, and 1900 with
// this).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0); }

__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// acc += A B^T over the 32-wide inner dimension (shared tiles, stride kLd).
// The 32 x 32 output is 4 x 4 blocks of 8 x 8; warp w owns row block w / 2
// and column blocks 2 (w % 2), 2 (w % 2) + 1. A fragment: A[row lane / 4][k +
// lane % 4]; B fragment: B[col lane / 4][k + lane % 4]; D fragment: row lane /
// 4, columns 2 (lane % 4) + {0, 1}.
__device__ __forceinline__ void mma_nt(const double* A, const double* B, double (&acc)[2][2]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ra = (warp >> 1) * 8 + (lane >> 2);
  const int cb0 = (warp & 1) * 16 + (lane >> 2);
  const int kq = lane & 3;
#pragma unroll
  for (int k0 = 0; k0 < kT; k0 += 4) {
    const double a = A[ra * kLd + k0 + kq];
    const double b0 = B[cb0 * kLd + k0 + kq];
    const double b1 = B[(cb0 + 8) * kLd + k0 + kq];
    dmma_8x8x4(acc[0], a, b0);
    dmma_8x8x4(acc[1], a, b1);
  }
}
__device__ __forceinline__ int frag_row() { return ((threadIdx.x >> 5) >> 1) * 8 + ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int frag_col(int blk) {
  return ((threadIdx.x >> 5) & 1) * 16 + blk * 8 + (threadIdx.x & 3) * 2;
}

// The two halves of a cluster barrier.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// This thread's global stores before bulk copies (async proxy) that other
// threads start after a barrier.
__device__ __forceinline__ void fence_stores_async() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
// Arrive on rank r's mbarrier: what this CTA wrote there before a barrier of its
// own is visible to whoever waits on it.
__device__ __forceinline__ void mbar_arrive_rank(uint64_t* bar, int r) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(saddr(bar)), "r"(r));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}

// 1 / d to within an ulp: the hardware approximation (rcp.approx.ftz.f64)
// refined by two Newton-Raphson steps x <- x + x (1 - d x), each of which
// squares the relative error. d is a positive normal pivot.
__device__ __forceinline__ double rcp_newton(double d) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  double e = fma(-d, x, 1.0);
  x = fma(x, e, x);
  e = fma(-d, x, 1.0);
  return fma(x, e, x);
}

// Warps 0 and 1: factor the symmetric tile in S.d (lower part used), LDL^T = Lu D
// Lu^T, and invert Lu: Lu below the diagonal of fac_lu(S) with D on it, Lu^-1 in
// fac_inv(S), sqrt(D) and its inverse in fac_sd(S). Four blocks of eight columns:
// the pivots by warp 0 (lane = row, the block in registers), then the columns right
// of it as 8 x 8 matrix products (each element the same chain of multiply-adds).
// After two blocks warp 1 inverts the first half, x = Lu11^-1, and forms z0 = e -
// Lu21 x while warp 0 goes on; last z = Lu22^-1 z0. The substitutions go column by
// column, each value into all later rows at once, so they are as deep as the block
// and not as its number of products. Few registers and little code: unrolled in two
// halves of 16 columns it took 15000 cycles a tile (25000 the first time, waiting
// for instructions), this 8000. What remains is the chain of the pivots, a
// reciprocal, a product and a multiply-add each. A non-positive pivot clears *ok
// and continues with pivot 1.
constexpr int kFs = kT + 1;
constexpr int kH = kT / 2;
__device__ __forceinline__ double* fac_lu(SolveSmem& S) { return S.ring[0]; }
__device__ __forceinline__ double* fac_inv(SolveSmem& S) { return S.ring[0] + kTS; }
__device__ __forceinline__ double* fac_sd(SolveSmem& S) { return S.ring[0] + 2 * kTS; }
__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// Unit lower triangular solve of 8 rows, column by column: v[r] -= t[r][m] v[m] for
// r > m, t at rows of kFs. SPLIT: the odd columns' products are summed apart, in s.
template <bool SPLIT>
__device__ __forceinline__ void tri8(const double* t, double (&v)[8], double (&s)[8]) {
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    if (SPLIT) v[m] += s[m];
#pragma unroll
    for (int r = m + 1; r < 8; ++r) {
      if (SPLIT && (m & 1))
        s[r] = fma(-t[r * kFs + m], v[m], s[r]);
      else
        v[r] = fma(-t[r * kFs + m], v[m], v[r]);
    }
  }
}

__device__ __noinline__ void factor_tile(SolveSmem& S, int* ok) {
  double* f = fac_lu(S);
  double* xs = fac_inv(S);
  double* sd = fac_sd(S);
  double* isd = sd + kT;
  double* u = sd + 2 * kT;    // 8 x 32: a block's columns before the division by their pivots
  double* odd = u + 8 * kT;   // 8 x kFs
  double* d = S.d;
  const int warp = warp_index(), lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
  int bad = 0;
  // One trailing 8 x 8 block (R, C) of d after the columns of block b.
  auto trail = [&](int b, int R, int C) {
    double* t = d + (R * 8 + lr) * kLd + C * 8 + 2 * lk;
    double c[2] = {t[0], t[1]};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = h * 4 + lk, p = b * 8 + k;
      const double l = f[(R * 8 + lr) * kFs + p];
      const bool half = b < 2 && C >= 2;  // across the halves: (l d) l, not l u
      dmma_8x8x4(c, half ? -l * f[p * kFs + p] : -l, half ? f[(C * 8 + lr) * kFs + p] : u[k * kT + C * 8 + lr]);
    }
    t[0] = c[0];
    t[1] = c[1];
  };
#pragma unroll 1
  for (int b = 0; b < 4; ++b) {
    if (warp == 0) {
      double a[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) a[m] = d[lane * kLd + b * 8 + m];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int pl = b * 8 + q;
        double p = __shfl_sync(0xffffffffu, a[q], pl);
        const double uq = a[q];
        u[q * kT + lane] = uq;
        double rp = rcp_newton(p);
        if (!(p > 0.0)) {  // beside the reciprocal, not before it
          bad = 1;
          p = rp = 1.0;
        }
        const double l = uq * rp;
        __syncwarp();
#pragma unroll
        for (int m = q + 1; m < 8; ++m) a[m] = fma(-l, u[q * kT + b * 8 + m], a[m]);
        f[lane * kFs + pl] = lane == pl ? p : l;
      }
      if (b == 3 && bad && lane == 0) *ok = 0;
    }
    if (b < 2) {
      pair_sync();
      // Block columns b + 1 .. 3, the rows dealt to both warps.
      for (int C = b + 1, n = 0; C < 4; ++C)
        for (int R = C; R < 4; ++R, ++n)
          if ((n & 1) == warp) trail(b, R, C);
      pair_sync();
      if (b == 1 && warp == 1) break;  // to the inverse of the first half
    } else if (b == 2) {
      __syncwarp();
      trail(2, 3, 3);
      __syncwarp();
    }
  }
  if (warp == 1) {
    // x = Lu11^-1, columns 0 .. 15, even and odd columns' products summed apart.
    double v[8], s[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      v[r] = r == lane ? 1.0 : 0.0;
      s[r] = 0.0;
    }
    tri8<true>(f, v, s);
#pragma unroll
    for (int r = 0; r < 8; ++r) xs[r * kFs + lane] = v[r];
    __syncwarp();
#pragma unroll
    for (int C = 0; C < 2; ++C)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int col = C * 8 + 2 * lk;
        double c[2] = {o == 0 && 8 + lr == col ? 1.0 : 0.0, o == 0 && 8 + lr == col + 1 ? 1.0 : 0.0};
        dmma_8x8x4(c, -f[(8 + lr) * kFs + 2 * lk + o], xs[(2 * lk + o) * kFs + C * 8 + lr]);
        double* t = o ? odd + lr * kFs : xs + (8 + lr) * kFs;
        t[col] = c[0];
        t[col + 1] = c[1];
      }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      v[r] = lane < kH ? xs[(8 + r) * kFs + lane] : 0.0;
      s[r] = lane < kH ? odd[r * kFs + lane] : 0.0;
    }
    tri8<true>(f + 8 * kFs + 8, v, s);
#pragma unroll
    for (int r = 0; r < 8; ++r) xs[(8 + r) * kFs + lane] = v[r];
    __syncwarp();
    // z0 = e - Lu21 x; columns c >= 16 are e_c.
#pragma unroll 1
    for (int R = 2; R < 4; ++R)
#pragma unroll
      for (int C = 0; C < 2; ++C) {
        double c[2] = {0.0, 0.0};
#pragma unroll
        for (int k0 = 0; k0 < kH; k0 += 4) dmma_8x8x4(c, -f[(R * 8 + lr) * kFs + k0 + lk], xs[(k0 + lk) * kFs + C * 8 + lr]);
        double* t = xs + (R * 8 + lr) * kFs + C * 8 + 2 * lk;
        t[0] = c[0];
        t[1] = c[1];
        t[kH] = R * 8 + lr == kH + C * 8 + 2 * lk ? 1.0 : 0.0;
        t[kH + 1] = R * 8 + lr == kH + C * 8 + 2 * lk + 1 ? 1.0 : 0.0;
      }
  }
  pair_sync();
  if (warp == 1) {
    // z = Lu22^-1 z0.
#pragma unroll 1
    for (int R = 2; R < 4; ++R) {
      double v[8], s[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = xs[(R * 8 + r) * kFs + lane];
      tri8<false>(f + R * 8 * kFs + R * 8, v, s);
#pragma unroll
      for (int r = 0; r < 8; ++r) xs[(R * 8 + r) * kFs + lane] = v[r];
      __syncwarp();
      if (R == 3) break;
#pragma unroll
      for (int C = 0; C < 4; ++C) {
        double* t = xs + (24 + lr) * kFs + C * 8 + 2 * lk;
        double c[2] = {t[0], t[1]};
#pragma unroll
        for (int k0 = 0; k0 < 8; k0 += 4)
          dmma_8x8x4(c, -f[(24 + lr) * kFs + kH + k0 + lk], xs[(kH + k0 + lk) * kFs + C * 8 + lr]);
        t[0] = c[0];
        t[1] = c[1];
      }
      __syncwarp();
    }
  } else {
    const double sq = sqrt(f[lane * kFs + lane]);
    sd[lane] = sq;
    isd[lane] = 1.0 / sq;
  }
  pair_sync();
}

// First column tile of E tile row c that can be non-zero: row 0 is rhs
// (dense); row e >= 1 is F^T row e - 1, non-zero only over its field block.
__device__ __forceinline__ int e_start(int c, int r, int k) {
  if (c == 0 || r == 0) return 0;
  return (((kT * c - 1) / r) * k) / kT;
}

// One system's operands and workspace.
struct Sys {
  double* A;           // lower tiles: L
  double* E;           // ne x nb tiles: appended rows
  double* Dv;          // nb tiles: inverses of the diagonal tiles
  const double* Mt;    // lower tiles of M
  const double* rhs;   // P
  const double* pen;   // k x k
  const double* fk;    // k x r
  double lam;
  int P, Pp, k, r, nfr, nb;
};

__device__ __forceinline__ double* a_tile(const Sys& y, int ti, int tj) {
  return y.A + static_cast<size_t>(tri_index(ti, tj)) * kTS;
}
__device__ __forceinline__ double* e_tile(const Sys& y, int c, int tj) {
  return y.E + static_cast<size_t>(c * y.nb + tj) * kTS;
}
__device__ __forceinline__ double* d_tile(const Sys& y, int j) { return y.Dv + static_cast<size_t>(j) * kTS; }

// Initial value of E (row, col): rhs in row 0, F^T below, zero padding.
__device__ __forceinline__ double e_init(const Sys& y, int row, int col) {
  if (row == 0) return col < y.P ? y.rhs[col] : 0.0;
  if (row > y.nfr) return 0.0;
  const int fb = (row - 1) / y.r, jj = (row - 1) - fb * y.r, m = col - fb * y.k;
  return (m >= 0 && m < y.k) ? y.fk[m * y.r + jj] : 0.0;
}

// Does A tile (ti, tj) hold an element of a diagonal field block (penalised)?
__device__ __forceinline__ bool a_pen_tile(const Sys& y, int ti, int tj) {
  const int r0 = ti * kT, c0 = tj * kT;
  if (r0 >= y.P || c0 >= y.P) return false;
  const int r1 = min(r0 + kT - 1, y.P - 1), c1 = min(c0 + kT - 1, y.P - 1);
  return max(r0 / y.k, c0 / y.k) <= min(r1 / y.k, c1 / y.k);
}

// Elements (r, c), (r, c + 1) of A tile (ti, tj) = M + lambda P0 (the penalty on the
// diagonal field blocks) before any update.
__device__ __forceinline__ void a_init2(const Sys& y, int ti, int tj, int r, int c, double (&out)[2]) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(y.Mt + static_cast<size_t>(tri_index(ti, tj)) * kTS + r * kLd + c));
  out[0] = v.x;
  out[1] = v.y;
  const int row = ti * kT + r;
  if (row >= y.P || !a_pen_tile(y, ti, tj)) return;
  const int rb = row / y.k;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int col = tj * kT + c + e, cm = col - rb * y.k;
    if (col < y.P && cm >= 0 && cm < y.k) out[e] = fma(y.lam, __ldg(y.pen + (row - rb * y.k) * y.k + cm), out[e]);
  }
}
// This thread's fragments of that tile, and of E tile (c, tj).
__device__ __forceinline__ void a_init(const Sys& y, int ti, int tj, double (&c)[2][2]) {
#pragma unroll
  for (int blk = 0; blk < 2; ++blk) a_init2(y, ti, tj, frag_row(), frag_col(blk), c[blk]);
}
__device__ __forceinline__ void e_frag(const Sys& y, int c, int tj, double (&v)[2][2]) {
#pragma unroll
  for (int blk = 0; blk < 2; ++blk)
#pragma unroll
    for (int e = 0; e < 2; ++e) v[blk][e] = e_init(y, c * kT + frag_row(), tj * kT + frag_col(blk) + e);
}

// Up to kGroup row tiles of one column that a CTA updates together.
struct Group {
  int n;                       // tiles
  const double* row[kGroup];   // tile (row, 0) of each: A or E
  int from[kGroup];            // first column tile that is not zero
};

// acc_u,q = L_q,p+u L_j,p+u^T for the U stages at buf, each product summed from
// zero over its 32 columns.
template <int N, int U>
__device__ __forceinline__ void group_products(const double* const (&buf)[U], double (&acc)[U][N][2][2]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ra = ((warp >> 1) * 8 + (lane >> 2)) * kLd + (lane & 3), rb = ((warp & 1) * 16 + (lane >> 2)) * kLd + (lane & 3);
#pragma unroll
  for (int k0 = 0; k0 < kT; k0 += 4)
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double b0 = buf[u][rb + k0], b1 = buf[u][rb + 8 * kLd + k0];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const double a = buf[u][(1 + q) * kTS + ra + k0];
        dmma_8x8x4(acc[u][q][0], a, b0);
        dmma_8x8x4(acc[u][q][1], a, b1);
      }
    }
}

// C_q = init_q - sum_p L_q,p L_j,p^T for p in [p0, p1) in order and the N row tiles
// of g. The operands of the next columns are in flight (stages of 1 + N tiles; lane
// 0 of warp 0 refills the stages of the step before once all warps have left them).
// A dependent FP64 matrix product comes back after some 160 cycles, ten times its
// issue, so few row tiles take several columns at once.
template <int N, class Init>
__device__ __forceinline__ void update_n(SolveSmem& S, unsigned& par, unsigned* status, int ring, const Group& g,
                                         const double* lj, int p0, int p1, double (&c)[kGroup][2][2], Init init) {
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int stages = min(ring / (1 + N), kStages);
  int load = p0, lst = 0;  // next column to load and its stage
  auto refill = [&](int upto, bool first) {
    for (; load < min(p1, upto); ++load) {
      if (!first && !mbar_wait(&S.empty[lst], ((par >> lst) & 1u) ^ 1u)) set_status(status, kStatusLoopLimit);
      if (lane == 0) {
        double* buf = S.ring[0] + lst * ((1 + N) * kTSz);
        uint32_t tiles = 1;
#pragma unroll
        for (int q = 0; q < N; ++q) tiles += load >= g.from[q];
        mbar_arrive_tx(&S.full[lst], tiles * kTileBytes);
        bulk_g2s(buf, lj + load * kTSz, kTileBytes, &S.full[lst]);
#pragma unroll
        for (int q = 0; q < N; ++q)
          if (load >= g.from[q]) bulk_g2s(buf + (1 + q) * kTS, g.row[q] + load * kTSz, kTileBytes, &S.full[lst]);
      }
      __syncwarp();
      lst = lst + 1 == stages ? 0 : lst + 1;
    }
  };
  if (warp == 0) {
    fence_proxy_async();
    refill(p0 + stages, true);
  }
  init();
  int p = p0, st = 0;
  auto step = [&](auto uc) {
    constexpr int U = decltype(uc)::value;
    if (warp == 0) refill(p + stages, false);
    const double* buf[U];
    int s_[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s_[u] = st;
      buf[u] = S.ring[0] + st * ((1 + N) * kTSz);
      if (!mbar_wait(&S.full[st], (par >> st) & 1u)) set_status(status, kStatusLoopLimit);
      par ^= 1u << st;
      st = st + 1 == stages ? 0 : st + 1;
    }
    double acc[U][N][2][2] = {};
    group_products<N, U>(buf, acc);
    __syncwarp();
    if (lane == 0)
#pragma unroll
      for (int u = 0; u < U; ++u) mbar_arrive(&S.empty[s_[u]]);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < N; ++q)
        if (p + u >= g.from[q])
#pragma unroll
          for (int e = 0; e < 4; ++e) c[q][e >> 1][e & 1] -= acc[u][q][e >> 1][e & 1];
    p += U;
  };
  if constexpr (N <= 2) {
    constexpr int U = N == 1 ? 4 : 2;
    while (p + U <= p1) step(std::integral_constant<int, U>{});
  }
  while (p < p1) step(std::integral_constant<int, 1>{});
  __syncthreads();  // the ring is free
}

template <class Init>
__device__ __forceinline__ void update_group(SolveSmem& S, unsigned& par, unsigned* status, int ring, const Group& g,
                                             const double* lj, int p0, int p1, double (&c)[kGroup][2][2], Init init) {
  int least = p1;
#pragma unroll
  for (int q = 0; q < kGroup; ++q)
    if (q < g.n) least = min(least, g.from[q]);
  p0 = max(p0, least);
  if (p0 >= p1) {
    init();
    return;
  }
  switch (g.n) {
    case 1: update_n<1>(S, par, status, ring, g, lj, p0, p1, c, init); break;
    case 2: update_n<2>(S, par, status, ring, g, lj, p0, p1, c, init); break;
    case 3: update_n<3>(S, par, status, ring, g, lj, p0, p1, c, init); break;
    case 4: update_n<4>(S, par, status, ring, g, lj, p0, p1, c, init); break;
  }
}

// The factoring rank's warps 2, 3, 6 and 7, off the schedulers of warps 0 and 1,
// which factor: the next diagonal tile's sum A_jj - sum_{p<p1} L_jp L_jp^T into
// `out`, its ten lower 8 x 8 blocks. Warps 2 and 6 share a scheduler, 3 and 7: five
// blocks to each pair (row 3's and row 0's, row 2's and row 1's).
__device__ __forceinline__ void diag_sum(SolveSmem& S, unsigned& par, unsigned* status, int ring, const Sys& y, int j,
                                         int p1, double* out) {
  const int warp = warp_index(), lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
  const int stages = min(ring - kRingStages, kStages);
  const double* row = a_tile(y, j, 0);
  double* ringp = S.ring[0] + kRingStages * kTSz;
  int load = 0, lst = 0;
  auto refill = [&](int upto, bool first) {
    for (; load < min(p1, upto); ++load) {
      if (!first && !mbar_wait(&S.empty[lst], ((par >> lst) & 1u) ^ 1u)) set_status(status, kStatusLoopLimit);
      if (lane == 0) {
        mbar_arrive_tx(&S.full[lst], kTileBytes);
        bulk_g2s(ringp + lst * kTSz, row + load * kTSz, kTileBytes, &S.full[lst]);
      }
      __syncwarp();
      lst = lst + 1 == stages ? 0 : lst + 1;
    }
  };
  if (warp == 2) {
    fence_proxy_async();
    refill(stages, true);
  }
  // Blocks (R, C): (3, 0) (3, 1) (3, 2) | (2, 0) (2, 1) (2, 2) | (3, 3) (0, 0) | (1, 0) (1, 1).
  constexpr int kMine = 3;
  const int n = warp < 4 ? 3 : 2;
  int R[kMine], C[kMine];
#pragma unroll
  for (int q = 0; q < kMine; ++q) {
    R[q] = warp == 2 ? 3 : warp == 3 ? 2 : warp == 6 ? (q == 0 ? 3 : 0) : 1;
    C[q] = warp == 6 ? (q == 0 ? 3 : 0) : q;
  }
  double c[kMine][2] = {};
#pragma unroll
  for (int q = 0; q < kMine; ++q)
    if (q < n) a_init2(y, j, j, R[q] * 8 + lr, C[q] * 8 + 2 * lk, c[q]);
  int st = 0;
  for (int p = 0; p < p1; ++p) {
    if (warp == 2) refill(p + stages, false);
    const double* t = ringp + st * kTSz + lr * kLd + lk;
    if (!mbar_wait(&S.full[st], (par >> st) & 1u)) set_status(status, kStatusLoopLimit);
    par ^= 1u << st;
    double acc[kMine][2] = {};
#pragma unroll
    for (int k0 = 0; k0 < kT; k0 += 4)
#pragma unroll
      for (int q = 0; q < kMine; ++q)
        if (q < n) dmma_8x8x4(acc[q], t[R[q] * 8 * kLd + k0], t[C[q] * 8 * kLd + k0]);
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.empty[st]);
#pragma unroll
    for (int q = 0; q < kMine; ++q) {
      c[q][0] -= acc[q][0];
      c[q][1] -= acc[q][1];
    }
    st = st + 1 == stages ? 0 : st + 1;
  }
#pragma unroll
  for (int q = 0; q < kMine; ++q)
    if (q < n) *reinterpret_cast<double2*>(out + (R[q] * 8 + lr) * kLd + C[q] * 8 + 2 * lk) = make_double2(c[q][0], c[q][1]);
}

__global__ void __launch_bounds__(kSolveThreads, 2) k_solve_cluster(SolveBatch b, int Pp, int Ep, size_t sys_stride, int ring, const double* __restrict__ Mt) {
  extern __shared__ __align__(16) unsigned char raw[];
  SolveSmem& S = *reinterpret_cast<SolveSmem*>(raw);
  const cg::cluster_group cl = cg::this_cluster();
  const int cn = static_cast<int>(cl.num_blocks());
  const int rank = static_cast<int>(cl.block_rank());
  const int s = blockIdx.x / cn;
  const int tid = threadIdx.x;
  Sys y;
  y.A = b.A + static_cast<size_t>(s) * sys_stride;
  const int nb = Pp / kT, ne = Ep / kT;
  y.nb = nb;
  y.E = y.A + static_cast<size_t>(nb * (nb + 1) / 2) * kTS;
  y.Dv = y.E + static_cast<size_t>(ne * nb) * kTS;
  y.P = b.P;
  y.Pp = Pp;
  y.k = b.k;
  y.r = b.r;
  y.nfr = b.nf * b.r;
  y.Mt = Mt + (b.m_index ? static_cast<size_t>(b.m_index[s]) * (nb * (nb + 1) / 2) * kTS : 0);
  y.rhs = b.rhs + (b.r_index ? static_cast<size_t>(b.r_index[s]) * y.P : 0);
  y.pen = b.pen;
  y.fk = b.fk;
  y.lam = b.lam[s];
  __shared__ int s_ok;
  __shared__ int s_estart[kMaxTiles];
  if (tid == 0) {
    s_ok = 1;
    auto init = [](uint64_t* bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(n) : "memory"); };
    for (int q = 0; q < kStages; ++q) {
      init(&S.full[q], 1);
      init(&S.empty[q], rank == 0 && cn > 1 ? 4 : kSolveThreads / 32);
    }
    init(&S.dbar, 1);
    init(&S.nbar, 1);
    init(&S.pbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int c = tid; c < ne; c += blockDim.x) s_estart[c] = e_start(c, y.r, y.k);
  __syncthreads();
  const int warp = warp_index(), ln = tid & 31, r0 = frag_row();
  // Rank 0 factors the diagonal tiles and takes no rows; a cluster of one does both.
  const bool solo = cn == 1, factors = rank == 0 && !solo;
  const int workers = solo ? 1 : cn - 1, wk = solo ? 0 : rank - 1;
  unsigned par = 0, dpar = 0, npar = 0;  // expected phase parities
  double tr = 0.0;                       // this thread's share of ||L^-1 F||^2
  Group g;
  double c[kGroup][2][2];
  auto rows_of = [&](int j) {  // row tiles of column j: below the diagonal, then E's active ones
    int n = 0;
    while (n < ne && s_estart[n] <= j) ++n;
    return nb - j - 1 + n;
  };
  // The group q0 .. of this worker's row tiles of column j, and their initial values.
  auto make_group = [&](int j, int q0) {
    const int below = nb - j - 1, nt = rows_of(j);
    g.n = 0;
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int t = wk + (q0 + q) * workers;
      if (t >= nt) break;
      g.n = q + 1;
      g.row[q] = t < below ? a_tile(y, j + 1 + t, 0) : e_tile(y, t - below, 0);
      g.from[q] = t < below ? 0 : s_estart[t - below];
    }
  };
  auto init_group = [&](int j, int q0) {
    const int below = nb - j - 1;
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int t = wk + (q0 + q) * workers;
      if (q >= g.n) break;
      if (t < below)
        a_init(y, j + 1 + t, j, c[q]);
      else
        e_frag(y, t - below, j, c[q]);
    }
  };
  // L_ij = C_ij Dinv_j^T for the group's tiles, stored; the squares of E's into tr.
  // L_{j+1,j} goes straight to the factoring rank as well.
  auto panel = [&](int j, int q0) {
#pragma unroll
    for (int q = 0; q < kGroup; ++q)
      if (q < g.n)
#pragma unroll
        for (int blk = 0; blk < 2; ++blk)
          *reinterpret_cast<double2*>(S.ring[0] + q * kTS + r0 * kLd + frag_col(blk)) = make_double2(c[q][blk][0], c[q][blk][1]);
    __syncthreads();
    if (!solo && q0 == 0) {
      if (!mbar_wait_cluster(&S.dbar, dpar)) set_status(b.status, kStatusLoopLimit);
      dpar ^= 1u;
      if (tid == 0) mbar_arrive_tx(&S.dbar, kTileBytes);  // the next one
    }
    const int below = nb - j - 1;
    const int ra = r0 * kLd + (ln & 3), rb = ((warp & 1) * 16 + (ln >> 2)) * kLd + (ln & 3);
#pragma unroll
    for (int q = 0; q < kGroup; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) c[q][e >> 1][e & 1] = 0.0;
#pragma unroll
    for (int k0 = 0; k0 < kT; k0 += 4) {
      const double b0 = S.d[rb + k0], b1 = S.d[rb + 8 * kLd + k0];
#pragma unroll
      for (int q = 0; q < kGroup; ++q)
        if (q < g.n) {
          const double a = S.ring[0][q * kTS + ra + k0];
          dmma_8x8x4(c[q][0], a, b0);
          dmma_8x8x4(c[q][1], a, b1);
        }
    }
    if (!solo && wk == 0 && q0 == 0 && below > 0) {
      double* nx = cl.map_shared_rank(&S.nx[0], 0);
#pragma unroll
      for (int blk = 0; blk < 2; ++blk)
        *reinterpret_cast<double2*>(nx + r0 * kLd + frag_col(blk)) = make_double2(c[0][blk][0], c[0][blk][1]);
      __syncthreads();
      if (tid == 0) mbar_arrive_rank(&S.nbar, 0);
    }
#pragma unroll
    for (int q = 0; q < kGroup; ++q)
      if (q < g.n) {
        const int t = wk + (q0 + q) * workers;
        double* out = const_cast<double*>(g.row[q]) + static_cast<size_t>(j) * kTS;
        const bool erow = t >= below && !(t == below && r0 == 0);
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          *reinterpret_cast<double2*>(out + r0 * kLd + frag_col(blk)) = make_double2(c[q][blk][0], c[q][blk][1]);
          if (erow) tr = fma(c[q][blk][0], c[q][blk][0], fma(c[q][blk][1], c[q][blk][1], tr));
        }
      }
    __syncthreads();
  };
  // L_jj and Dinv_j = D^-1/2 Lu^-1 from factor_tile's parts: to the workspace, and
  // Dinv_j to `keep`.
  auto publish = [&](int j, double* keep) {
    const double *f = fac_lu(S), *xs = fac_inv(S), *sd = fac_sd(S), *isd = sd + kT;
    const int r = tid >> 3, c0 = (tid & 7) * 4;
    double l[4], d[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      l[e] = c0 + e < r ? f[r * kFs + c0 + e] * sd[c0 + e] : (c0 + e == r ? sd[r] : 0.0);
      d[e] = xs[r * kFs + c0 + e] * isd[r];
    }
    auto put = [&](double* t, const double (&v)[4]) {
      reinterpret_cast<double2*>(t + r * kLd + c0)[0] = make_double2(v[0], v[1]);
      reinterpret_cast<double2*>(t + r * kLd + c0)[1] = make_double2(v[2], v[3]);
    };
    put(keep, d);
    if (!solo) {
      fence_proxy_async();
      __syncthreads();
      if (tid == 0)
        for (int w = 1; w < cn; ++w) bulk_s2rank(S.d, keep, kTileBytes, &S.dbar, w);
    }
    put(a_tile(y, j, j), l);
    put(d_tile(y, j), d);
  };
  auto frag_put = [&](double* t, const double (&v)[2][2]) {
#pragma unroll
    for (int blk = 0; blk < 2; ++blk)
      *reinterpret_cast<double2*>(t + r0 * kLd + frag_col(blk)) = make_double2(v[blk][0], v[blk][1]);
  };

  // Column by column, left-looking: C_ij = A_ij - sum_{p<j} L_ip L_jp^T stays in
  // registers and is stored once, as L_ij. One cluster barrier per column says that
  // column j is stored; between its two halves the ranks sum column j + 1 up to
  // p < j, then take p = j. Dinv_j (rank 0 to all) and L_{j+1,j} (rank 1 to rank 0),
  // which the chain from one diagonal tile to the next passes through, go straight
  // to the other rank's shared memory and are signalled on its mbarrier.
  if (!solo) {
    if (!factors && tid == 0) mbar_arrive_tx(&S.dbar, kTileBytes);
    cluster_arrive();
  }
  if (factors) {
    double *dinv = S.ring[0] + kRingDinv * kTSz, *sum = S.ring[0] + kRingDiag * kTSz, *prev = S.ring[0] + kRingPrev * kTSz;
    unsigned ppar = 0;
    a_init(y, 0, 0, c[0]);
    for (int j = 0; j < nb; ++j) {
      if (j > 0) {
        // The sum up to p < j - 2 is there (diag_sum).
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const double2 v = *reinterpret_cast<const double2*>(sum + r0 * kLd + frag_col(blk));
          c[0][blk][0] = v.x;
          c[0][blk][1] = v.y;
        }
        for (int last = j > 1 ? 0 : 1; last < 2; ++last) {
          if (last == 0) {
            if (!mbar_wait(&S.pbar, ppar)) set_status(b.status, kStatusLoopLimit);
            ppar ^= 1u;
          } else {
            if (!mbar_wait_cluster(&S.nbar, npar)) set_status(b.status, kStatusLoopLimit);
            npar ^= 1u;
          }
          const double* t = last ? S.nx : prev;
          double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
          mma_nt(t, t, acc);
#pragma unroll
          for (int e = 0; e < 4; ++e) c[0][e >> 1][e & 1] -= acc[e >> 1][e & 1];
        }
      }
      frag_put(S.d, c[0]);
      __syncthreads();
      if (warp < 2)
        factor_tile(S, &s_ok);
      else if ((warp & 2) != 0 && j + 1 < nb)
        diag_sum(S, par, b.status, ring, y, j + 1, j - 1, sum);
      cluster_wait();  // column j - 1 is stored, and Dinv_{j-1} no longer read
      __syncthreads();
      publish(j, dinv);
      if (tid == 0 && j > 0 && j + 1 < nb) {
        mbar_arrive_tx(&S.pbar, kTileBytes);
        bulk_g2s(prev, a_tile(y, j + 1, j - 1), kTileBytes, &S.pbar);
      }
      cluster_arrive();
    }
  } else {
    enum { kDiag, kRows, kTail };
    int mode = solo ? kDiag : kRows;
    for (int j = 0, q0 = 0;;) {
      int p0 = 0, p1 = j;
      if (mode == kDiag) {
        g.n = 1;
        g.row[0] = a_tile(y, j, 0);
        g.from[0] = 0;
      } else if (mode == kRows) {
        make_group(j, q0);
        if (!solo && q0 == 0) p1 = j - 1;
      } else {
        p0 = j - 1;
      }
      update_group(S, par, b.status, ring, g, a_tile(y, j, 0), p0, p1, c, [&] {
        if (mode == kDiag)
          a_init(y, j, j, c[0]);
        else if (mode == kRows)
          init_group(j, q0);
      });
      if (mode == kDiag) {
        frag_put(S.d, c[0]);
        __syncthreads();
        if (warp < 2) factor_tile(S, &s_ok);
        __syncthreads();
        publish(j, S.d);
        __syncthreads();
        mode = kRows;
        continue;
      }
      if (!solo && q0 == 0 && mode == kRows) {
        cluster_wait();  // column j - 1 is stored
        mode = kTail;
        continue;
      }
      panel(j, q0);
      q0 += kGroup;
      mode = kRows;
      if (wk + q0 * workers < rows_of(j)) continue;
      q0 = 0;
      fence_stores_async();
      if (solo) {
        __syncthreads();
        mode = kDiag;
      } else {
        cluster_arrive();
      }
      if (++j == nb) break;
    }
  }
  if (!solo) cluster_wait();

  // Trace partial of this rank (fixed-order tree), then rank 0 finishes.
  S.red[tid] = tr;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (tid < o) S.red[tid] += S.red[tid + o];
    __syncthreads();
  }
  if (tid == 0) b.partial[static_cast<size_t>(s) * cn + rank] = S.red[0];
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;
  if (tid == 0) {
    double t2 = 0.0;
    for (int q = 0; q < cn; ++q) t2 += b.partial[static_cast<size_t>(s) * cn + q];
    if (b.want_edf) b.edf[s] = static_cast<double>(y.P) - y.lam * t2;
    b.ok[s] = s_ok;
  }
  // theta = L^-T y, y = E row 0: column tiles from the last, each
  // theta_i = Dinv_i^T y_i, then y_q -= L_iq^T theta_i for q < i. While warp 0 forms
  // theta_i from Dinv_i in shared memory, each thread has its first column of L_i
  // and its part of the next Dinv on the way.
  double* v = S.ring[0];
  for (int q = tid; q < Pp; q += blockDim.x) v[q] = __ldcg(e_tile(y, 0, q >> 5) + (q & 31));
  const int dr = (tid >> 3) * kLd + (tid & 7) * 4;
  auto dinv_at = [&](int i) { return S.ring[0] + (1 + (i & 1)) * kTSz; };
  auto put_dinv = [&](int i, const double2 (&d)[2]) {
    reinterpret_cast<double2*>(dinv_at(i) + dr)[0] = d[0];
    reinterpret_cast<double2*>(dinv_at(i) + dr)[1] = d[1];
  };
  auto get_dinv = [&](int i, double2 (&d)[2]) {
    const double2* t = reinterpret_cast<const double2*>(d_tile(y, i) + dr);
    d[0] = __ldcg(t);
    d[1] = __ldcg(t + 1);
  };
  double2 dn[2];
  get_dinv(nb - 1, dn);
  put_dinv(nb - 1, dn);
  __syncthreads();
  for (int i = nb - 1; i >= 0; --i) {
    auto column = [&](int q) { return a_tile(y, i, q >> 5) + (q & 31); };
    double lc[kT];
    if (i > 0) get_dinv(i - 1, dn);
    if (tid < i * kT) {
      const double* c = column(tid);
#pragma unroll
      for (int r = 0; r < kT; ++r) lc[r] = __ldcg(c + r * kLd);
    }
    if (warp == 0) {
      const double* D = dinv_at(i);
      double t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int r = 0; r < kT; r += 2) {
        t0 = fma(D[r * kLd + ln], v[i * kT + r], t0);
        t1 = fma(D[(r + 1) * kLd + ln], v[i * kT + r + 1], t1);
      }
      __syncwarp();
      v[i * kT + ln] = t0 + t1;
    }
    __syncthreads();
    for (int q = tid; q < i * kT; q += blockDim.x) {
      if (q != tid) {
        const double* c = column(q);
#pragma unroll
        for (int r = 0; r < kT; ++r) lc[r] = __ldcg(c + r * kLd);
      }
      double a0 = v[q], a1 = 0.0;
#pragma unroll
      for (int r = 0; r < kT; r += 2) {
        a0 = fma(-lc[r], v[i * kT + r], a0);
        a1 = fma(-lc[r + 1], v[i * kT + r + 1], a1);
      }
      v[q] = a0 + a1;
    }
    if (i > 0) put_dinv(i - 1, dn);
    __syncthreads();
  }
  for (int q = tid; q < y.P; q += blockDim.x) b.theta[static_cast<size_t>(s) * y.P + q] = v[q];
}

// About two CTAs per SM over the batch, at most the portable cluster size 8. Sixteen
// to a cluster (more than a device must offer, so the launch asks) where each CTA
// still has an SM to itself and there are row tiles for the workers: one system of
// 736 unknowns with its penalty rows takes 420 us and not 590, five without 340 and
// not 390; ten, two CTAs on an SM, 470 and not 395.
constexpr int kMaxRanks = 16;
int solve_cluster_size(int nsys, int rows) {
  if (rows >= 12 && nsys * kMaxRanks <= 148) return kMaxRanks;
  const int want = std::min(8, std::max(1, (148 * 2) / std::max(nsys, 1)));
  int cn = 1;
  while (cn * 2 <= want) cn *= 2;
  return cn;
}

// The lower tiles of each distinct M in the tile-major layout, identity
// padding outside P x P (grid: tiles x matrices).
__global__ void __launch_bounds__(256) k_solve_prep(const double* __restrict__ M, int P, double* __restrict__ Mt) {
  const int u = blockIdx.x, m = blockIdx.y;
  int ti = static_cast<int>((sqrtf(8.0f * static_cast<float>(u) + 1.0f) - 1.0f) * 0.5f);
  if (tri_index(ti + 1, 0) <= u) ++ti;
  if (tri_index(ti, 0) > u) --ti;
  const int tj = u - tri_index(ti, 0);
  const double* Mm = M + static_cast<size_t>(m) * P * P;
  double* dst = Mt + (static_cast<size_t>(m) * gridDim.x + u) * kTS;
  for (int e = threadIdx.x; e < kT * kT; e += blockDim.x) {
    const int r = e >> 5, c = e & 31, row = ti * kT + r, col = tj * kT + c;
    dst[r * kLd + c] = (row < P && col < P) ? Mm[static_cast<size_t>(row) * P + col] : (row == col ? 1.0 : 0.0);
  }
}

void launch_solve_batch(Context& c, const SolveBatch& b) {
  const int Pp = solve_pp(b.P);
  const int Ep = solve_ep(b.nf, b.r);
  if (b.P > 1024) fail(DGPU_ERR_INVALID, "solve: more than 1024 unknowns is not supported");
  if (Ep / kT > kMaxTiles) fail(DGPU_ERR_INVALID, "solve: penalty factor too wide");
  if (b.k > 1024 || b.r > b.k) fail(DGPU_ERR_INVALID, "solve: penalty factor shape is not supported");
  if (b.nsys <= 0) return;
  const int nb = Pp / kT, nm = std::max(b.nm, 1);
  const size_t sys_stride = solve_sys_doubles(b.P, b.nf, b.r);
  double* Mt = b.A + static_cast<size_t>(b.nsys) * sys_stride;
  k_solve_prep<<<dim3(static_cast<unsigned>(nb * (nb + 1) / 2), static_cast<unsigned>(nm)), 256, 0, c.stream>>>(b.M, b.P, Mt);
  DGPU_LAUNCH("k_solve_prep");
  int cn = solve_cluster_size(b.nsys, nb - 1 + Ep / kT);
  const void* kernel = reinterpret_cast<const void*>(k_solve_cluster);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  int ring = 0;
  auto configure = [&] {
    ring = b.nsys * cn <= 148 ? kRingLarge : kRingSmall;
    const size_t smem = solve_smem(ring);
    ensure_dynamic_smem(kernel, smem);
    cfg.gridDim = dim3(static_cast<unsigned>(b.nsys * cn));
    cfg.blockDim = dim3(kSolveThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cn);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  };
  configure();
  if (cn > 8) {
    if (c.solve_ranks16 < 0) {
      int most = 0;
      const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                      cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) == cudaSuccess && most > 0;
      if (!ok) cudaGetLastError();
      c.solve_ranks16 = ok ? 1 : 0;
    }
    if (c.solve_ranks16 == 0) {
      cn = 8;
      configure();
    }
  }
  SolveBatch bb = b;
  DGPU_CUDA(cudaLaunchKernelEx(&cfg, k_solve_cluster, bb, Pp, Ep, sys_stride, ring, static_cast<const double*>(Mt)));
  DGPU_LAUNCH("k_solve_cluster");
  // Systems whose Cholesky met a non-positive pivot are redone by pivoted
  // LDL^T, as the reference falls back from LLT to LDLT (src/solve.cpp:177-181).
  if (b.skip_ldlt) return;
  StageTimer t(c, "fit: LDLT fallback");
  launch_ldlt_fallback(c, b);
}

// out = A_s^{-1} v = L^-T (L^-1 v) from system s's factor tiles, one CTA.
// The tiles are first pulled into L2 (one bulk prefetch per tile; streaming
// kernels that ran since the solve may have evicted them) and, up to 24 tile
// columns, every Dinv tile into shared memory. Forward over the column tiles:
// y_i = Dinv_i y_i (warp 0), then y_p -= L_pi y_i for the rows below (a thread
// per row); backward: theta_i = Dinv_i^T y_i, then y_q -= L_iq^T theta_i (a
// thread per column). Each thread's first row (column) of the next step is
// loaded into registers while the current step finishes, so the L2 latency
// overlaps the step's barriers and the diagonal solve.
constexpr int kAiThreads = 512;
constexpr int kDs = kT * (kT + 1);  // one Dinv tile in shared memory, padded rows
constexpr int kAiPreloadTiles = 24;

int apply_inverse_smem(int nb) { return static_cast<int>(sizeof(double)) * kDs * (nb <= kAiPreloadTiles ? nb : 1); }

__device__ __forceinline__ void ai_row(const double* __restrict__ A, int tile, int rr, double (&v)[kT]) {
  const double2* src = reinterpret_cast<const double2*>(A + static_cast<size_t>(tile) * kTS + rr * kLd);
#pragma unroll
  for (int c = 0; c < kT / 2; ++c) {
    const double2 t = __ldg(src + c);
    v[2 * c] = t.x;
    v[2 * c + 1] = t.y;
  }
}

__device__ __forceinline__ void ai_col(const double* __restrict__ A, int tile, int cc, double (&v)[kT]) {
  const double* src = A + static_cast<size_t>(tile) * kTS + cc;
#pragma unroll
  for (int r = 0; r < kT; ++r) v[r] = __ldg(src + r * kLd);
}

__global__ void __launch_bounds__(kAiThreads) k_apply_inverse(const double* __restrict__ A, const double* __restrict__ Dv,
                                                               int P, int Pp, const double* __restrict__ vin,
                                                               double* __restrict__ out) {
  extern __shared__ double dsm[];  // Dinv tiles (all, or the current one)
  __shared__ double y[1024];
  const int tid = threadIdx.x, warp = tid >> 5, ln = tid & 31;
  const int nb = Pp / kT, na = nb * (nb + 1) / 2;
  const bool all = nb <= kAiPreloadTiles;
  for (int u = tid; u < na + nb; u += blockDim.x) {
    const double* tile = u < na ? A + static_cast<size_t>(u) * kTS : Dv + static_cast<size_t>(u - na) * kTS;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(tile), "r"(static_cast<unsigned>(kTS * 8)) : "memory");
  }
  for (int q = tid; q < Pp; q += blockDim.x) y[q] = q < P ? vin[q] : 0.0;
  if (all)
    for (int e = tid; e < nb * kT * kT; e += blockDim.x) {
      const int t = e / (kT * kT), rc = e - t * (kT * kT);
      dsm[t * kDs + (rc >> 5) * (kT + 1) + (rc & 31)] = Dv[static_cast<size_t>(t) * kTS + (rc >> 5) * kLd + (rc & 31)];
    }
  double lv[kT];
  {
    const int p = kT + tid;
    if (p < Pp) ai_row(A, tri_index(p >> 5, 0), p & 31, lv);
  }
  __syncthreads();
  for (int i = 0; i < nb; ++i) {
    const double* D = dsm + (all ? i * kDs : 0);
    if (!all) {
      const double* Dg = Dv + static_cast<size_t>(i) * kTS;
      for (int e = tid; e < kT * kT; e += blockDim.x) dsm[(e >> 5) * (kT + 1) + (e & 31)] = Dg[(e >> 5) * kLd + (e & 31)];
      __syncthreads();
    }
    if (warp == 0) {
      double t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int c = 0; c < kT; c += 2) {
        t0 = fma(D[ln * (kT + 1) + c], y[i * kT + c], t0);
        t1 = fma(D[ln * (kT + 1) + c + 1], y[i * kT + c + 1], t1);
      }
      __syncwarp();
      y[i * kT + ln] = t0 + t1;
    }
    __syncthreads();
    const int p = (i + 1) * kT + tid;
    if (p < Pp) {
      double a0 = y[p], a1 = 0.0;
#pragma unroll
      for (int c = 0; c < kT / 2; ++c) {
        a0 = fma(-lv[2 * c], y[i * kT + 2 * c], a0);
        a1 = fma(-lv[2 * c + 1], y[i * kT + 2 * c + 1], a1);
      }
      y[p] = a0 + a1;
    }
    for (int p2 = p + kAiThreads; p2 < Pp; p2 += kAiThreads) {
      double l2[kT];
      ai_row(A, tri_index(p2 >> 5, i), p2 & 31, l2);
      double a0 = y[p2], a1 = 0.0;
#pragma unroll
      for (int c = 0; c < kT / 2; ++c) {
        a0 = fma(-l2[2 * c], y[i * kT + 2 * c], a0);
        a1 = fma(-l2[2 * c + 1], y[i * kT + 2 * c + 1], a1);
      }
      y[p2] = a0 + a1;
    }
    const int pn = (i + 2) * kT + tid;  // this thread's first row of the next step
    if (i + 1 < nb && pn < Pp) ai_row(A, tri_index(pn >> 5, i + 1), pn & 31, lv);
    __syncthreads();
  }
  {
    const int q = tid;
    if (nb > 1 && q < (nb - 1) * kT) ai_col(A, tri_index(nb - 1, q >> 5), q & 31, lv);
  }
  for (int i = nb - 1; i >= 0; --i) {
    if (warp == 0) {
      double t0 = 0.0, t1 = 0.0;
      if (all) {
        const double* D = dsm + i * kDs;
#pragma unroll
        for (int r = 0; r < kT; r += 2) {
          t0 = fma(D[r * (kT + 1) + ln], y[i * kT + r], t0);
          t1 = fma(D[(r + 1) * (kT + 1) + ln], y[i * kT + r + 1], t1);
        }
      } else {
        const double* D = Dv + static_cast<size_t>(i) * kTS;
#pragma unroll
        for (int r = 0; r < kT; r += 2) {
          t0 = fma(D[r * kLd + ln], y[i * kT + r], t0);
          t1 = fma(D[(r + 1) * kLd + ln], y[i * kT + r + 1], t1);
        }
      }
      __syncwarp();
      y[i * kT + ln] = t0 + t1;
    }
    __syncthreads();
    const int q = tid;
    if (q < i * kT) {
      double a0 = y[q], a1 = 0.0;
#pragma unroll
      for (int r = 0; r < kT; r += 2) {
        a0 = fma(-lv[r], y[i * kT + r], a0);
        a1 = fma(-lv[r + 1], y[i * kT + r + 1], a1);
      }
      y[q] = a0 + a1;
    }
    for (int q2 = q + kAiThreads; q2 < i * kT; q2 += kAiThreads) {
      double c2[kT];
      ai_col(A, tri_index(i, q2 >> 5), q2 & 31, c2);
      double a0 = y[q2], a1 = 0.0;
#pragma unroll
      for (int r = 0; r < kT; r += 2) {
        a0 = fma(-c2[r], y[i * kT + r], a0);
        a1 = fma(-c2[r + 1], y[i * kT + r + 1], a1);
      }
      y[q2] = a0 + a1;
    }
    if (i >= 1 && q < (i - 1) * kT) ai_col(A, tri_index(i - 1, q >> 5), q & 31, lv);
    __syncthreads();
  }
  for (int q = tid; q < P; q += blockDim.x) out[q] = y[q];
}

void launch_apply_inverse(cudaStream_t st, const SolveBatch& b, int s, const double* v, double* out) {
  const int Pp = solve_pp(b.P), nb = Pp / kT, ne = solve_ep(b.nf, b.r) / kT;
  const double* A = b.A + static_cast<size_t>(s) * solve_sys_doubles(b.P, b.nf, b.r);
  const double* Dv = A + static_cast<size_t>(nb * (nb + 1) / 2 + ne * nb) * kTS;
  const int smem = apply_inverse_smem(nb);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_apply_inverse), smem);
  k_apply_inverse<<<1, kAiThreads, smem, st>>>(A, Dv, b.P, Pp, v, out);
  DGPU_LAUNCH("k_apply_inverse");
}

}  // namespace dgpu
