// Gradient of the stamp fit's GCV score (reference src/solve.cpp:147-193,
// GCV = n RSS / (n - edf)^2) and of its weighted residual sum of squares RSS,
// with respect to log lambda, the kernel shift (dx, dy) and the scale s, by the
// adjoint of the normal-equation map. No reference counterpart.
//
// The stamp rows are X_row = u(row) (x) d(row) (u_c = s B_n,c for c < nc, the
// B_n convolved with the shifted basis; u_nc = 1 for the background; d the
// thin-plate design row), M = X^T W X, b = X^T W t, A = M + lambda P0 with
// P0 = F F^T, theta = A^-1 b, H = A^-1 F. With g = dRSS/dtheta = -2 lambda P0 theta
// and z = A^-1 g = -2 lambda H (F^T theta):
//   dRSS/dM = theta theta^T - sym(z theta^T),  dRSS/db = -2 theta + z,
//   dedf/dM = lambda H H^T,                   dedf/db = 0,
//   dGCV = alpha dRSS + beta dedf,  alpha = n/(n-edf)^2, beta = 2 n RSS/(n-edf)^3,
//   dRSS/dlambda = 2 lambda (F^T theta)^T (F^T H) (F^T theta),
//   dedf/dlambda = -tr(F^T H) + lambda ||F^T H||_F^2.
// Back through X: Xbar = 2 W X Mbar + W t bbar^T, and per row
// Ubar_c = sum_j d_j Xbar_(c,j); then dx += sum_c Ubar_c dU_c/ddx with
// dU_c/ddx = -s B^x_n,c (the B_n of the x-derivative taps), dy alike, and
// ds += sum_c Ubar_c u_c / s. The H H^T part is one product over all rows (see
// k_gcv_edf).
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "fit_internal.h"
#include "gcv_grad_internal.h"

namespace dgpu {

// B = [rhs | F] (P x (1 + nf r)), F = blockdiag(fk) over the nf fields.
__global__ void k_build_rhs_f(int P, int k, int r, const double* __restrict__ rhs, const double* __restrict__ fk,
                              double* __restrict__ B) {
  const int m = 1 + (P / k) * r;
  const int64_t n = static_cast<int64_t>(P) * m;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(e / m), col = static_cast<int>(e - static_cast<int64_t>(p) * m);
    double v;
    if (col == 0) {
      v = rhs[p];
    } else {
      const int q = col - 1, fb = q / r, i = q - fb * r;
      v = (p / k == fb) ? fk[(p % k) * r + i] : 0.0;
    }
    B[e] = v;
  }
}

// theta (column 0 of X) contiguous; ftheta_q = f_q . theta.
__global__ void k_theta_ftheta(int P, int k, int r, const double* __restrict__ X, const double* __restrict__ fk,
                               double* __restrict__ theta, double* __restrict__ ftheta) {
  const int m = 1 + (P / k) * r;
  for (int p = threadIdx.x; p < P; p += blockDim.x) theta[p] = X[static_cast<size_t>(p) * m];
  for (int q = threadIdx.x; q < m - 1; q += blockDim.x) {
    const int fb = q / r, i = q - fb * r;
    double s = 0.0;
    for (int j = 0; j < k; ++j) s = fma(fk[j * r + i], X[static_cast<size_t>(fb * k + j) * m], s);
    ftheta[q] = s;
  }
}

// Row q of G = F^T H: stats[q] = {G_qq, sum_q' G_qq'^2, ftheta_q * (G ftheta)_q}.
__global__ void k_fth_rows(int P, int k, int r, const double* __restrict__ X, const double* __restrict__ fk,
                           const double* __restrict__ ftheta, double* __restrict__ stats) {
  const int m = 1 + (P / k) * r, nq = m - 1;
  const int q = blockIdx.x, fb = q / r, i = q - fb * r;
  __shared__ double red[3][32];
  double sq = 0.0, gf = 0.0, diag = 0.0;
  for (int q2 = threadIdx.x; q2 < nq; q2 += blockDim.x) {
    double g = 0.0;
    for (int j = 0; j < k; ++j) g = fma(fk[j * r + i], X[static_cast<size_t>(fb * k + j) * m + 1 + q2], g);
    sq = fma(g, g, sq);
    gf = fma(g, ftheta[q2], gf);
    if (q2 == q) diag = g;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
    gf += __shfl_xor_sync(0xffffffffu, gf, o);
    diag += __shfl_xor_sync(0xffffffffu, diag, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][warp] = diag;
    red[1][warp] = sq;
    red[2][warp] = gf;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
    stats[static_cast<size_t>(q) * 3 + threadIdx.x] = threadIdx.x == 2 ? t * ftheta[q] : t;
  }
}

// z = -2 lambda H ftheta.
__global__ void k_zvec(int P, int k, int r, const double* __restrict__ X, const double* __restrict__ ftheta, double lam,
                       double* __restrict__ z) {
  const int m = 1 + (P / k) * r;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  double s = 0.0;
  for (int q = 0; q < m - 1; ++q) s = fma(X[static_cast<size_t>(p) * m + 1 + q], ftheta[q], s);
  z[p] = -2.0 * lam * s;
}

// GCV scalars from the fixed-order sums. sums = {trace G, ||G||^2, ftheta^T G ftheta};
// raw = ywy - 2 theta.b + theta^T M theta; n rows.
__global__ void k_gcv_scalars(int P, double lam, const double* __restrict__ sums, const double* __restrict__ raw,
                              const long long* __restrict__ n, GcvScalars* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double nn = static_cast<double>(*n);
  double rss = *raw;
  if (rss < 0.0) rss = 0.0;
  const double edf = static_cast<double>(P) - lam * sums[0];
  const double den = nn - edf;
  GcvScalars s;
  s.rss = rss;
  s.edf = edf;
  s.n = nn;
  s.gcv = den > 0.0 ? nn * rss / (den * den) : __longlong_as_double(0x7ff0000000000000ll);
  s.alpha = den > 0.0 ? nn / (den * den) : 0.0;
  s.beta = den > 0.0 ? 2.0 * nn * rss / (den * den * den) : 0.0;
  const double drss = 2.0 * lam * sums[2];
  const double dedf = -sums[0] + lam * sums[1];
  s.drss_dloglam = lam * drss;
  s.dgcv_dloglam = lam * (s.alpha * drss + s.beta * dedf);
  s.lam = lam;
  *out = s;
}

constexpr int kGrRows = 128;  // rows (threads) per block
constexpr int kGrMaxK = 32;

// RSS part, a thread per row. Per block: {alpha dRSS/ddx, ddy, ds, dRSS/ddx, ddy, ds}
// over its rows.
__global__ void __launch_bounds__(kGrRows) k_gcv_rows(GcvRowsArgs a) {
  extern __shared__ __align__(16) double gsm[];
  const int nc = a.nc, nf = nc + 1, k = a.k, P = nf * k;
  double* st = gsm;    // theta
  double* sz = st + P;  // z
  const int tid = threadIdx.x;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kGrRows + tid;
  const bool live = row < a.N && a.valid[row] && a.w[row] > 0.0;
  const GcvScalars S = *a.scal;
  const double wr = live ? a.w[row] : 0.0, tr = live ? a.t[row] : 0.0;
  for (int p = tid; p < P; p += kGrRows) {
    st[p] = a.theta[p];
    sz[p] = a.z[p];
  }
  double d[kGrMaxK];
#pragma unroll
  for (int j = 0; j < kGrMaxK; ++j) d[j] = (live && j < k) ? a.d[row * k + j] : 0.0;
  __syncthreads();
  double g[6] = {0, 0, 0, 0, 0, 0};
  const double inv_s = 1.0 / a.scale;
  if (live) {
    const double* bn = a.bn + row * nc;
    const double* bnx = a.bnx + row * nc;
    const double* bny = a.bny + row * nc;
    auto dots = [&](int c, double& dt, double& dz) {
      dt = dz = 0.0;
#pragma unroll
      for (int j = 0; j < kGrMaxK; ++j)
        if (j < k) {
          dt = fma(d[j], st[c * k + j], dt);
          dz = fma(d[j], sz[c * k + j], dz);
        }
    };
    // X theta and X z.
    double xt = 0.0, xz = 0.0;
    for (int c = 0; c < nf; ++c) {
      double dt, dz;
      dots(c, dt, dz);
      const double u = c < nc ? bn[c] : 1.0;
      xt = fma(u, dt, xt);
      xz = fma(u, dz, xz);
    }
    for (int c = 0; c < nc; ++c) {
      double dt, dz;
      dots(c, dt, dz);
      // RSS part (alpha = 1): 2 w (X Mbar)_c + w t bbar_c, d-contracted.
      const double ur = 2.0 * wr * (xt * dt - 0.5 * (xz * dt + xt * dz)) + wr * tr * (-2.0 * dt + dz);
      const double u = bn[c], bx = bnx[c], by = bny[c];
      g[3] -= ur * bx;
      g[4] -= ur * by;
      g[5] += ur * u * inv_s;
      const double ug = S.alpha * ur;
      g[0] -= ug * bx;
      g[1] -= ug * by;
      g[2] += ug * u * inv_s;
    }
  }
  // Fixed-order block reduction.
  __shared__ double red[6][kGrRows / 32];
  for (int i = 0; i < 6; ++i) {
    double v = g[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[i][tid >> 5] = v;
  }
  __syncthreads();
  if (tid < 6) {
    double t = 0.0;
    for (int w = 0; w < kGrRows / 32; ++w) t += red[tid][w];
    a.partial[static_cast<size_t>(blockIdx.x) * 6 + tid] = t;
  }
}

// ---------------------------------------------------------------------------
// edf part of the GCV gradient.
//
// Per row, with K = H H^T and S_cc' = sum_mm' K_(c,m)(c',m') d_m d_m' (symmetric
// in c, c'), the row's share of dedf/ddx is -2 w beta lambda sum_cc' bx_c S_cc' u_c'.
// S over all rows is one product of the rows' design pairs V[i][{m,m'}] =
// d_m d_m' (k (k+1) / 2 wide) with the packed Kp[{m,m'}][{c,c'}], so it runs on
// the FP64 tensor cores and each S value is used where it is made: it meets
// the weights of its pair (bx_c u_c' + bx_c' u_c for dx, alike for dy and the
// scale) in the epilogue and is not stored. Contracting each row with the
// nf r columns of H instead (X_row h_q, then its d-contraction) takes 3.5 times
// the products on the vector pipe: 22.9 ms at 1.9e5 rows, P = 464; this way
// 1.35 ms, bound by the DMMA pipe (13 GFMA with padding, 0.72 ms at 37 TFLOP/s).
//
// A CTA takes 128 rows x 16 NT pairs of components, eight warps of 32 x 8 NT,
// the design pairs in chunks of 16: V is generated into one buffer while the
// tensor cores read the other; Kp (zero padded) arrives by cp.async.
// ---------------------------------------------------------------------------
constexpr int kGeK = 16;             // design pairs per chunk
constexpr int kGeLa = kGrRows + 4;   // row strides = 4 mod 16 doubles: conflict-free fragment loads

__host__ __device__ inline int ge_pairs(int n) { return n * (n + 1) / 2; }
__host__ __device__ inline int ge_pad(int n, int to) { return (n + to - 1) / to * to; }

// (a, b), a <= b, of the idx-th pair in row-major order over the upper triangle of n.
__device__ __forceinline__ int2 pair_of(int idx, int n) {
  int a = 0, left = n;
  while (idx >= left) {
    idx -= left;
    ++a;
    --left;
  }
  return make_int2(a, a + idx);
}

__device__ __forceinline__ void dmma_gcv(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// K = H H^T (P x P), H the last nq columns of X (row stride m = nq + 1): a
// 32 x 32 tile per CTA of four warps.
__global__ void __launch_bounds__(128) k_hht(int P, int m, const double* __restrict__ X, double* __restrict__ K) {
  __shared__ double A[32][36], B[32][36];
  const int p0 = blockIdx.x * 32, q0 = blockIdx.y * 32, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, q = lane >> 2, kq = lane & 3;
  const int wr = (warp >> 1) * 16, wc = (warp & 1) * 16;
  double acc[2][2][2] = {};
  for (int c0 = 1; c0 < m; c0 += 32) {
    __syncthreads();
    for (int e = tid; e < 32 * 32; e += 128) {
      const int r = e >> 5, c = e & 31;
      A[r][c] = (p0 + r < P && c0 + c < m) ? X[static_cast<size_t>(p0 + r) * m + c0 + c] : 0.0;
      B[r][c] = (q0 + r < P && c0 + c < m) ? X[static_cast<size_t>(q0 + r) * m + c0 + c] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 4) {
      const double a0 = A[wr + q][k0 + kq], a1 = A[wr + 8 + q][k0 + kq];
      const double b0 = B[wc + q][k0 + kq], b1 = B[wc + 8 + q][k0 + kq];
      dmma_gcv(acc[0][0], a0, b0);
      dmma_gcv(acc[0][1], a0, b1);
      dmma_gcv(acc[1][0], a1, b0);
      dmma_gcv(acc[1][1], a1, b1);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = p0 + wr + 8 * i + q, c = q0 + wc + 8 * j + 2 * kq + e;
        if (r < P && c < P) K[static_cast<size_t>(r) * P + c] = acc[i][j][e];
      }
}

// Kp[{m,m'}][{c,c'}] (vp x sp, zero padded): K_(c,m)(c',m') + K_(c,m')(c',m), once when m = m'.
__global__ void __launch_bounds__(128) k_pack_k(int nf, int k, int sp, const double* __restrict__ K,
                                                double* __restrict__ kp) {
  const int v = blockIdx.x, P = nf * k;
  const int2 mm = v < ge_pairs(k) ? pair_of(v, k) : make_int2(-1, -1);
  for (int s = threadIdx.x; s < sp; s += blockDim.x) {
    double x = 0.0;
    if (mm.x >= 0 && s < ge_pairs(nf)) {
      const int2 cc = pair_of(s, nf);
      x = K[static_cast<size_t>(cc.x * k + mm.x) * P + cc.y * k + mm.y];
      if (mm.x != mm.y) x += K[static_cast<size_t>(cc.x * k + mm.y) * P + cc.y * k + mm.x];
    }
    kp[static_cast<size_t>(v) * sp + s] = x;
  }
}

template <int NT>
__host__ __device__ constexpr int ge_lb() { return 16 * NT + 4; }
// Main loop: 2 x V chunk, 2 x Kp chunk, the rows' design values (k x 128), the
// pair table; epilogue, in the same memory: u, bx, by (nc x 128 each).
template <int NT>
size_t ge_smem(int nc, int k) {
  const size_t main = sizeof(double) * (2 * kGeK * (kGeLa + ge_lb<NT>()) + static_cast<size_t>(k) * kGeLa) +
                      sizeof(int2) * ge_pad(ge_pairs(k), kGeK);
  return std::max(main, sizeof(double) * 3 * nc * kGeLa);
}

template <int NT>
__global__ void __launch_bounds__(256, 2) k_gcv_edf(GcvRowsArgs a, const double* __restrict__ kp, int sp, int vp,
                                                    double* __restrict__ part) {
  extern __shared__ __align__(16) double gsm[];
  constexpr int LB = ge_lb<NT>();
  const int nc = a.nc, nf = nc + 1, k = a.k;
  double* As = gsm;                        // 2 x kGeK x kGeLa
  double* Bs = As + 2 * kGeK * kGeLa;      // 2 x kGeK x LB
  double* sd = Bs + 2 * kGeK * LB;         // k x kGeLa
  int2* pt = reinterpret_cast<int2*>(sd + k * kGeLa);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, kq = lane & 3;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kGrRows;
  const int s0 = blockIdx.y * 16 * NT;
  const int myrow = tid & (kGrRows - 1);
  auto live_row = [&](int r) { return row0 + r < a.N && a.valid[row0 + r] && a.w[row0 + r] > 0.0; };
  auto load_b = [&](int v0, int buf) {
    for (int e = tid; e < kGeK * 8 * NT; e += 256) {  // 16-byte pieces
      const int r = e / (8 * NT), c = 2 * (e - r * 8 * NT);
      const double* src = kp + static_cast<size_t>(v0 + r) * sp + s0 + c;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(
                       __cvta_generic_to_shared(Bs + (buf * kGeK + r) * LB + c))), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_b(0, 0);
  for (int e = tid; e < kGrRows * k; e += 256) {
    const int r = e / k, j = e - r * k;
    sd[j * kGeLa + r] = live_row(r) ? a.d[(row0 + r) * k + j] : 0.0;
  }
  for (int v = tid; v < vp; v += 256) pt[v] = v < ge_pairs(k) ? pair_of(v, k) : make_int2(-1, -1);
  __syncthreads();
  auto gen = [&](int v0, int buf) {
    const int h = (tid >> 7) * (kGeK / 2);
#pragma unroll
    for (int j = 0; j < kGeK / 2; ++j) {
      const int2 p = pt[v0 + h + j];
      As[(buf * kGeK + h + j) * kGeLa + myrow] = p.x >= 0 ? sd[p.x * kGeLa + myrow] * sd[p.y * kGeLa + myrow] : 0.0;
    }
  };
  gen(0, 0);
  double acc[4][NT][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 8 * NT;
  int buf = 0;
  for (int v0 = 0; v0 < vp; v0 += kGeK, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // this chunk is in place; the other buffers are read
    if (v0 + kGeK < vp) {
      load_b(v0 + kGeK, buf ^ 1);
      gen(v0 + kGeK, buf ^ 1);
    }
#pragma unroll
    for (int k0 = 0; k0 < kGeK; k0 += 4) {
      const double* A = As + (buf * kGeK + k0 + kq) * kGeLa + wm + q;
      const double* B = Bs + (buf * kGeK + k0 + kq) * LB + wn + q;
      double af[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) af[i] = A[8 * i];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const double bf = B[8 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i) dmma_gcv(acc[i][j], af[i], bf);
      }
    }
  }
  __syncthreads();
  double* su = gsm;  // nc x kGeLa each
  double* sx = su + nc * kGeLa;
  double* sy = sx + nc * kGeLa;
  for (int e = tid; e < kGrRows * nc; e += 256) {
    const int r = e / nc, c = e - r * nc;
    const bool live = live_row(r);
    const int64_t at = (row0 + r) * nc + c;
    su[c * kGeLa + r] = live ? a.bn[at] : 0.0;
    sx[c * kGeLa + r] = live ? a.bnx[at] : 0.0;
    sy[c * kGeLa + r] = live ? a.bny[at] : 0.0;
  }
  __syncthreads();
  double g[3] = {0.0, 0.0, 0.0};
  double rx[4] = {}, ry[4] = {}, rs[4] = {};
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int s = s0 + wn + 8 * j + 2 * kq + e;
      if (s >= ge_pairs(nf)) continue;
      const int2 cc = pair_of(s, nf);
      if (cc.x >= nc) continue;  // the background with itself: no kernel component
      const double* p0 = su + cc.x * kGeLa + wm + q;
      const int step = nc * kGeLa;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double v = acc[i][j][e];
        const double u0 = p0[8 * i], x0 = p0[step + 8 * i], y0 = p0[2 * step + 8 * i];
        if (cc.y == nc) {  // u_c' = 1, no component
          rx[i] = fma(v, x0, rx[i]);
          ry[i] = fma(v, y0, ry[i]);
          rs[i] = fma(v, u0, rs[i]);
        } else if (cc.x == cc.y) {
          rx[i] = fma(v, x0 * u0, rx[i]);
          ry[i] = fma(v, y0 * u0, ry[i]);
          rs[i] = fma(v, u0 * u0, rs[i]);
        } else {
          const double* p1 = su + cc.y * kGeLa + wm + q;
          const double u1 = p1[8 * i], x1 = p1[step + 8 * i], y1 = p1[2 * step + 8 * i];
          rx[i] = fma(v, fma(x0, u1, x1 * u0), rx[i]);
          ry[i] = fma(v, fma(y0, u1, y1 * u0), ry[i]);
          rs[i] = fma(v, 2.0 * u0 * u1, rs[i]);
        }
      }
    }
  const GcvScalars S = *a.scal;
  const double inv_s = 1.0 / a.scale;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = wm + 8 * i + q;
    const double coef = live_row(r) ? 2.0 * a.w[row0 + r] * S.beta * S.lam : 0.0;
    g[0] = fma(-coef, rx[i], g[0]);
    g[1] = fma(-coef, ry[i], g[1]);
    g[2] = fma(coef * inv_s, rs[i], g[2]);
  }
  __shared__ double red[3][8];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double v = g[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[i][warp] = v;
  }
  __syncthreads();
  if (tid < 3) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[tid][w];
    part[(static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * 3 + tid] = t;
  }
}

// out6 = the column sums of the row partials, plus the edf partials in the
// first three (fixed order: lanes stride the rows, then a shuffle tree).
__global__ void __launch_bounds__(192) k_gcv_sum(const double* __restrict__ part, int nrows,
                                                 const double* __restrict__ edf, int nedf, double* __restrict__ out6) {
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double t = 0.0;
  for (int r = lane; r < nrows; r += 32) t += part[static_cast<size_t>(r) * 6 + i];
  if (i < 3)
    for (int r = lane; r < nedf; r += 32) t += edf[static_cast<size_t>(r) * 3 + i];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) out6[i] = t;
}

// Fixed-order column sums (one thread per column, rows in order).
__global__ void k_colsum(const double* __restrict__ part, int nrows, int ncols, double* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  double t = 0.0;
  for (int r = 0; r < nrows; ++r) t += part[static_cast<size_t>(r) * ncols + c];
  out[c] = t;
}

int gcv_rhs_cols(int P, int k, int r) { return 1 + (P / k) * r; }

void launch_build_rhs_f(cudaStream_t st, int P, int k, int r, const double* rhs, const double* fk, double* B) {
  const int64_t n = static_cast<int64_t>(P) * gcv_rhs_cols(P, k, r);
  k_build_rhs_f<<<static_cast<int>(std::min<int64_t>((n + 255) / 256, 1184)), 256, 0, st>>>(P, k, r, rhs, fk, B);
  DGPU_LAUNCH("k_build_rhs_f");
}

void launch_gcv_theta(cudaStream_t st, int P, int k, int r, const double* X, const double* fk, double* work) {
  const int nq = gcv_rhs_cols(P, k, r) - 1;
  k_theta_ftheta<<<1, 512, 0, st>>>(P, k, r, X, fk, work, work + P);
  DGPU_LAUNCH("k_theta_ftheta");
  (void)nq;
}

void launch_gcv_stats(cudaStream_t st, int P, int k, int r, const double* X, const double* fk, double lam,
                      const double* raw, const long long* n, double* work, GcvScalars* scal) {
  const int nq = gcv_rhs_cols(P, k, r) - 1;
  double* theta = work;
  double* ftheta = theta + P;
  double* z = ftheta + nq;
  double* stats = z + P;
  double* sums = stats + 3 * static_cast<size_t>(nq);
  (void)theta;
  k_fth_rows<<<nq, 256, 0, st>>>(P, k, r, X, fk, ftheta, stats);
  DGPU_LAUNCH("k_fth_rows");
  k_colsum<<<1, 32, 0, st>>>(stats, nq, 3, sums);
  DGPU_LAUNCH("k_colsum");
  k_zvec<<<(P + 127) / 128, 128, 0, st>>>(P, k, r, X, ftheta, lam, z);
  DGPU_LAUNCH("k_zvec");
  k_gcv_scalars<<<1, 32, 0, st>>>(P, lam, sums, raw, n, scal);
  DGPU_LAUNCH("k_gcv_scalars");
}

size_t gcv_stats_doubles(int P, int k, int r) {
  const int nq = gcv_rhs_cols(P, k, r) - 1;
  return 2 * static_cast<size_t>(P) + 4 * static_cast<size_t>(nq) + 8;
}

namespace {
int gcv_rows_blocks(int64_t N) { return static_cast<int>((N + kGrRows - 1) / kGrRows); }
// Pairs of components per CTA: the width with the least padding, the wider one on a tie.
int ge_nt(int nf) { return ge_pad(ge_pairs(nf), 96) <= ge_pad(ge_pairs(nf), 48) ? 6 : 3; }
}  // namespace

size_t gcv_rows_doubles(int64_t N, int nc, int k) {
  const int nf = nc + 1, bn = 16 * ge_nt(nf);
  const size_t P = static_cast<size_t>(nf) * k, sp = ge_pad(ge_pairs(nf), bn), vp = ge_pad(ge_pairs(k), kGeK);
  return P * P + sp * vp + (6 + 3 * sp / bn) * static_cast<size_t>(gcv_rows_blocks(N)) + 2;
}

void launch_gcv_rows(cudaStream_t st, const GcvRowsArgs& a, double* work, double* out6) {
  if (a.k > kGrMaxK) fail(DGPU_ERR_INVALID, "stamp_gcv: at most 32 knots are supported");
  const int nf = a.nc + 1, P = nf * a.k;
  if (sizeof(double) * (8 * static_cast<size_t>(P) + 3 * static_cast<size_t>(a.nc) * kGrRows) > 200 * 1024)
    fail(DGPU_ERR_INVALID, "stamp_gcv: basis too large for the row contraction");
  const int nt = ge_nt(nf), bn = 16 * nt, nb = gcv_rows_blocks(a.N);
  const int sp = ge_pad(ge_pairs(nf), bn), vp = ge_pad(ge_pairs(a.k), kGeK);
  double* kp = work;  // 16-byte rows for cp.async: first, sp is a multiple of 48
  double* K = kp + static_cast<size_t>(sp) * vp;
  double* edf = K + static_cast<size_t>(P) * P;
  GcvRowsArgs r = a;
  r.partial = edf + 3 * static_cast<size_t>(sp / bn) * nb;
  k_hht<<<dim3((P + 31) / 32, (P + 31) / 32), 128, 0, st>>>(P, a.nq + 1, a.X, K);
  DGPU_LAUNCH("k_hht");
  k_pack_k<<<vp, 128, 0, st>>>(nf, a.k, sp, K, kp);
  DGPU_LAUNCH("k_pack_k");
  const size_t smem = sizeof(double) * 2 * static_cast<size_t>(P);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_gcv_rows), smem);
  k_gcv_rows<<<nb, kGrRows, smem, st>>>(r);
  DGPU_LAUNCH("k_gcv_rows");
  auto go = [&](auto kern, size_t bytes) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(kern), bytes);
    kern<<<dim3(nb, sp / bn), 256, bytes, st>>>(a, kp, sp, vp, edf);
  };
  if (nt == 6)
    go(k_gcv_edf<6>, ge_smem<6>(a.nc, a.k));
  else
    go(k_gcv_edf<3>, ge_smem<3>(a.nc, a.k));
  DGPU_LAUNCH("k_gcv_edf");
  k_gcv_sum<<<1, 192, 0, st>>>(r.partial, nb, edf, (sp / bn) * nb, out6);
  DGPU_LAUNCH("k_gcv_sum");
}

}  // namespace dgpu
