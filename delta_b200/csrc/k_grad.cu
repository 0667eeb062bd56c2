// Weighted chi^2 of the spatially varying kernel model and its adjoints.
//
// The model is the subtraction's (src/subtract.cpp:466-639) with two more
// parameters, a sub-pixel shift d = (dx, dy) of the kernel and a photometric
// scale s:
//   M(x) = s * sum_c a_c(x) C_c(x) + b(x),   C_c = K_c^d (*) R~,
//   K_c^d(u, v) = g_nx(u - dx) g_ny(v - dy),
// with the reference sanitised as the subtraction does (masked / non-finite
// pixels -> the fill value, off-frame -> 0) and a_c, b blended from the coarse
// lattice of theta. The objective is chi^2 = sum_x W(x) (S(x) - M(x))^2 over
// pixels with W > 0 and a finite S.
//
// k_chi2_tile (one CTA per 32 x 16 output tile) recomputes, from the staged
// reference window, the x passes with g and g' and the y passes of every
// component for C_c, C^x_c = g'_nx g_ny (*) R~ and C^y_c = g_nx g'_ny (*) R~
// (so dC_c/ddx = -C^x_c, dC_c/ddy = -C^y_c): the N_basis convolved images are
// never stored. Per pixel, with rbar = -2 W (S - M):
//   dchi2/ds   += rbar sum_c a_c C_c
//   dchi2/ddx  -= rbar s sum_c a_c C^x_c     (dy alike)
//   q_c(x)      = rbar s C_c (c < nc),  q_nc = rbar   (dchi2/da_c(x))
// chi^2 and the scalar gradients are reduced per CTA in FP64 and summed in a
// fixed order. C_c (c < nc), rbar and p = rbar s are written out for the adjoints.
// k_grad_tile.cu holds the same tiles for the common basis shapes; this kernel
// serves the others (n_max 0, 1, 7, 8; fewer than 9 or more than 40 taps).
//
// k_theta_grad: dchi2/dtheta_{c,j} = sum_x q_c(x) D_j(x), where D_j(x) is the
// same lattice blend applied to the j-th design function (the fields of the
// identity theta): the adjoint of the lattice evaluation and blend.
//
// k_adjoint_reference: dchi2/dR(y) = sum_c sum_u K_c^d(u) p(y + u) a_c(y + u)
// with p = rbar s: the correlation of the field-weighted residual with the
// flipped kernel field, zero where the reference was replaced by the fill
// value (which is held constant).
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "grad_internal.h"

namespace dgpu {

constexpr int kGTW = 32;  // tile width
constexpr int kGTH = 16;  // tile height
constexpr int kGThreads = 256;

namespace {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

size_t chi2_tile_smem(int n_max, int ks) {
  const int kh = (ks - 1) / 2, nx = n_max + 1;
  const int nrows = kGTH + 2 * kh, wcols = kGTW + 2 * kh;
  return sizeof(float) * (static_cast<size_t>(nrows) * wcols + 2 * static_cast<size_t>(nx) * nrows * kGTW +
                          4 * static_cast<size_t>(nx) * ks);
}

__global__ void __launch_bounds__(kGThreads) k_chi2_tile(Chi2Args a) {
  extern __shared__ __align__(16) float smem[];
  const int ks = a.ks, kh = (ks - 1) / 2, nx = a.n_max + 1;
  const int nrows = kGTH + 2 * kh, wcols = kGTW + 2 * kh;
  float* win = smem;                                        // nrows x wcols
  float* tx = win + nrows * wcols;                          // nx x nrows x 32: g_nx (*)_x R~
  float* tdx = tx + nx * nrows * kGTW;                      // nx x nrows x 32: g'_nx (*)_x R~
  float* gx = tdx + nx * nrows * kGTW;                      // nx x ks
  float* dgx = gx + nx * ks;
  float* gy = dgx + nx * ks;
  float* dgy = gy + nx * ks;
  const int bx = blockIdx.x * kGTW, by = blockIdx.y * kGTH, tid = threadIdx.x;
  const int w = a.w, h = a.h;
  const float fill = *a.fill;
  for (int i = tid; i < nx * ks; i += blockDim.x) {
    gx[i] = a.gx[i];
    dgx[i] = a.dgx[i];
    gy[i] = a.gy[i];
    dgy[i] = a.dgy[i];
  }
  for (int i = tid; i < nrows * wcols; i += blockDim.x) {
    const int r = i / wcols, c = i - r * wcols;
    const int yy = by - kh + r, xx = bx - kh + c;
    float v = 0.0f;
    if (yy >= 0 && yy < h && xx >= 0 && xx < w) {
      const size_t idx = static_cast<size_t>(yy) * w + xx;
      v = __ldg(a.ref + idx);
      if ((a.rmask && __ldg(a.rmask + idx) != 0) || !isfinite(v)) v = fill;
    }
    win[i] = v;
  }
  __syncthreads();
  // x passes: tx[q][r][lx] = sum_j g_q[j] R~[r][lx + 2kh - j] (and tdx with g').
  for (int it = tid; it < nrows * kGTW; it += blockDim.x) {
    const int r = it / kGTW, lx = it - r * kGTW;
    const float* row = win + r * wcols + lx + 2 * kh;
    float acc[kGradMaxNx], accd[kGradMaxNx];
#pragma unroll
    for (int q = 0; q < kGradMaxNx; ++q) acc[q] = accd[q] = 0.0f;
    for (int j = 0; j < ks; ++j) {
      const float v = row[-j];
#pragma unroll
      for (int q = 0; q < kGradMaxNx; ++q) {
        if (q < nx) {
          acc[q] = fmaf(gx[q * ks + j], v, acc[q]);
          accd[q] = fmaf(dgx[q * ks + j], v, accd[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kGradMaxNx; ++q) {
      if (q < nx) {
        tx[(q * nrows + r) * kGTW + lx] = acc[q];
        tdx[(q * nrows + r) * kGTW + lx] = accd[q];
      }
    }
  }
  __syncthreads();
  double chi = 0.0, g_s = 0.0, g_dx = 0.0, g_dy = 0.0;
  const int lx = tid % kGTW;
  const float s = a.scale;
  const size_t N = static_cast<size_t>(w) * h;
  for (int ly = tid / kGTW; ly < kGTH; ly += kGThreads / kGTW) {
    const int x = bx + lx, y = by + ly;
    if (x >= w || y >= h) continue;
    const size_t idx = static_cast<size_t>(y) * w + x;
    float m0 = 0.0f, mx = 0.0f, my = 0.0f;
    float cv[kGradMaxNc];  // C_c of this pixel, kept for q
    // per component: C, C^x, C^y at (lx, ly): buffer row ly + 2kh - j.
    for (int c = 0; c < a.nc; ++c) {
      const int2 o = a.orders[c];
      const float* col = tx + (o.x * nrows + ly + 2 * kh) * kGTW + lx;
      const float* cold = tdx + (o.x * nrows + ly + 2 * kh) * kGTW + lx;
      const float* g = gy + o.y * ks;
      const float* dg = dgy + o.y * ks;
      float cc = 0.0f, cx = 0.0f, cy = 0.0f;
      for (int j = 0; j < ks; ++j) {
        const float t = col[-j * kGTW];
        cc = fmaf(g[j], t, cc);
        cy = fmaf(dg[j], t, cy);
        cx = fmaf(g[j], cold[-j * kGTW], cx);
      }
      const float ac = field_point(a.F, c, x, y);
      m0 = fmaf(ac, cc, m0);
      mx = fmaf(ac, cx, mx);
      my = fmaf(ac, cy, my);
      cv[c] = cc;
    }
    const float bg = field_point(a.F, a.nc, x, y);
    const float model = fmaf(s, m0, bg);
    const float sv = __ldg(a.sci + idx);
    const float wt = __ldg(a.weight + idx);
    const bool ok = wt > 0.0f && isfinite(sv) && isfinite(model);
    const float r = ok ? sv - model : 0.0f;
    const float rb = ok ? -2.0f * wt * r : 0.0f;
    if (ok) {
      chi += static_cast<double>(wt) * static_cast<double>(r) * static_cast<double>(r);
      g_s += static_cast<double>(rb) * static_cast<double>(m0);
      g_dx -= static_cast<double>(rb) * static_cast<double>(s) * static_cast<double>(mx);
      g_dy -= static_cast<double>(rb) * static_cast<double>(s) * static_cast<double>(my);
    }
    if (a.q) {
      for (int c = 0; c < a.nc; ++c) a.q[static_cast<size_t>(c) * N + idx] = cv[c];
      a.q[static_cast<size_t>(a.nc) * N + idx] = rb;
    }
    if (a.p) a.p[idx] = rb * s;
  }
  // Fixed-order block reduction of the four sums.
  __shared__ double red[4][kGThreads / 32];
  chi = warp_sum_d(chi);
  g_s = warp_sum_d(g_s);
  g_dx = warp_sum_d(g_dx);
  g_dy = warp_sum_d(g_dy);
  const int warp = tid >> 5;
  if ((tid & 31) == 0) {
    red[0][warp] = chi;
    red[1][warp] = g_s;
    red[2][warp] = g_dx;
    red[3][warp] = g_dy;
  }
  __syncthreads();
  if (tid < 4) {
    double t = 0.0;
    for (int i = 0; i < kGThreads / 32; ++i) t += red[tid][i];
    a.partial[static_cast<size_t>(blockIdx.y * gridDim.x + blockIdx.x) * 4 + tid] = t;
  }
}

// out[c] = sum over rows r of part[r * ncols + c], a CTA per column: threads
// stride the rows, then a fixed tree. (One thread per column over the 8192 tiles
// of a 2048^2 frame was a 0.4 ms chain of dependent loads.)
__global__ void __launch_bounds__(256) k_sum_rows(const double* __restrict__ part, int nrows, int ncols,
                                                  double* __restrict__ out) {
  __shared__ double red[8];
  double t = 0.0;
  for (int r = threadIdx.x; r < nrows; r += 256) t += part[static_cast<size_t>(r) * ncols + blockIdx.x];
  t = warp_sum_d(t);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    t = 0.0;
    for (int i = 0; i < 8; ++i) t += red[i];
    out[blockIdx.x] = t;
  }
}

// sum_x q_f(x) D_j(x) on the FP64 tensor cores: fields x design functions with
// the pixels as the inner dimension, exact products of float32 values. A warp
// takes 32 pixels at a time, lane = pixel: the planes of the next 32 arrive by
// cp.async (coalesced, one plane per instruction) while it blends D, brings both
// into the fragment layout through shared memory and multiplies; q_c = p C_c is
// rounded to float32 as it is read. One tile of 32 fields x 8 NT design
// functions per CTA (blockIdx.y, .z), its warps' sums added in order. Floor:
// reading the planes (nf + 1 floats per pixel: 0.5 GB at 2048^2, 29 fields, 75 us
// at 6.5 TB/s). One FP64 FMA chain per thread and pair took 1.53 ms, this 0.22 ms.
constexpr int kTgWarps = 8;
constexpr int kTgLd = 36;  // conflict-free fragments

__device__ __forceinline__ void dmma_grad(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// One float to shared memory, 0 when !in (src is then not read).
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(in ? 4 : 0)
               : "memory");
}

template <int NT>
__global__ void __launch_bounds__(kTgWarps * 32, 2)
k_theta_grad(int w, int h, int nf, int k, const float* __restrict__ q, const float* __restrict__ p, DevFields D,
             double* __restrict__ part) {
  extern __shared__ __align__(16) float sm[];
  constexpr int NJ = 8 * NT, kBuf = 33 * kTgLd, kWarpFloats = 2 * kBuf + NJ * kTgLd;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, kq = lane & 3;
  float* sq = sm + warp * kWarpFloats;  // 2 x (32 planes, then p) x kTgLd
  float* sd = sq + 2 * kBuf;            // NJ x kTgLd
  const int f0 = blockIdx.z * 32, j0 = blockIdx.y * NJ, nfl = min(32, nf - f0), nj = min(NJ, k - j0);
  const int nc = nf - 1 - f0;           // planes below nc are C_c (times p), plane nc is rbar
  const int64_t N = static_cast<int64_t>(w) * h;
  for (int i = lane; i < kWarpFloats; i += 32) sq[i] = 0.0f;  // planes past the last stay zero
  __syncwarp();
  auto load = [&](int64_t b, int buf) {
    const int64_t px = min(b + lane, N - 1);
    const bool in = b + lane < N;
    float* dst = sq + buf * kBuf + lane;
    const float* src = q + static_cast<size_t>(f0) * N + px;
    for (int f = 0; f < nfl; ++f) cp_async4(dst + f * kTgLd, src + static_cast<size_t>(f) * N, in);
    cp_async4(dst + 32 * kTgLd, p + px, in);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[4][NT][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kTgWarps * 32;
  int64_t b = (static_cast<int64_t>(blockIdx.x) * kTgWarps + warp) * 32;
  if (b < N) load(b, 0);
  for (int buf = 0; b < N; b += step, buf ^= 1) {
    if (b + step < N) load(b + step, buf ^ 1);
    const int64_t px = min(b + lane, N - 1);
    const int y = static_cast<int>(px / w), x = static_cast<int>(px - static_cast<int64_t>(y) * w);
    if (D.exact) {
      for (int j = 0; j < nj; ++j) sd[j * kTgLd + lane] = __ldg(D.full + static_cast<size_t>(j0 + j) * N + px);
    } else {
      const size_t plane = static_cast<size_t>(D.ncx) * D.ncy;
      const float* c0 = D.latf + j0 * plane + static_cast<size_t>(D.celly[y]) * D.ncx + D.cellx[x];
      const float fy = D.wy[y], wx = D.wx[x];
#pragma unroll 8
      for (int j = 0; j < nj; ++j, c0 += plane)
        sd[j * kTgLd + lane] = cell_blend(__ldg(c0), __ldg(c0 + 1), __ldg(c0 + D.ncx), __ldg(c0 + D.ncx + 1), fy, wx);
    }
    if (b + step < N)
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    else
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    const float* cur = sq + buf * kBuf;
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 4) {
      const float pv = cur[32 * kTgLd + k0 + kq];
      double bf[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j) bf[j] = static_cast<double>(sd[(8 * j + r) * kTgLd + k0 + kq]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float v = cur[(8 * i + r) * kTgLd + k0 + kq];
        const double af = static_cast<double>(8 * i + r < nc ? pv * v : v);
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma_grad(acc[i][j], af, bf[j]);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  double* red = reinterpret_cast<double*>(sm);  // warps x 32 x NJ
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) red[(warp * 32 + 8 * i + r) * NJ + 8 * j + 2 * kq + e] = acc[i][j][e];
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * NJ; e += kTgWarps * 32) {
    const int f = e / NJ, j = e - f * NJ;
    if (f0 + f >= nf || j0 + j >= k) continue;
    double t = 0.0;
    for (int i = 0; i < kTgWarps; ++i) t += red[i * 32 * NJ + e];
    part[static_cast<size_t>(blockIdx.x) * nf * k + (f0 + f) * k + j0 + j] = t;
  }
}

size_t adjoint_ref_smem(int ks) {
  const int kh = (ks - 1) / 2;
  const int nrows = kGTH + 2 * kh, wcols = kGTW + 2 * kh;
  return sizeof(float) * (2 * static_cast<size_t>(nrows) * wcols + static_cast<size_t>(nrows) * kGTW);
}

// rbar_R(y) = sum_c sum_{u,v} g_nx(u - dx) g_ny(v - dy) (p a_c)(y + (u, v)), p = rbar s.
__global__ void __launch_bounds__(kGThreads) k_adjoint_reference(AdjRefArgs a) {
  extern __shared__ __align__(16) float smem[];
  const int ks = a.ks, kh = (ks - 1) / 2;
  const int nrows = kGTH + 2 * kh, wcols = kGTW + 2 * kh;
  float* pw = smem;                  // p over the window
  float* pc = pw + nrows * wcols;    // p * a_c over the window
  float* xb = pc + nrows * wcols;    // x correlation, nrows x 32
  const int bx = blockIdx.x * kGTW, by = blockIdx.y * kGTH, tid = threadIdx.x;
  const int w = a.w, h = a.h;
  for (int i = tid; i < nrows * wcols; i += blockDim.x) {
    const int r = i / wcols, c = i - r * wcols;
    const int yy = by - kh + r, xx = bx - kh + c;
    pw[i] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? a.p[static_cast<size_t>(yy) * w + xx] : 0.0f;
  }
  float out[kGTH / (kGThreads / kGTW)];
  constexpr int kRows = kGTH / (kGThreads / kGTW);
  for (int i = 0; i < kRows; ++i) out[i] = 0.0f;
  const int lx = tid % kGTW, ly0 = tid / kGTW;
  for (int c = 0; c < a.nc; ++c) {
    const int2 o = a.orders[c];
    __syncthreads();
    for (int i = tid; i < nrows * wcols; i += blockDim.x) {
      const int r = i / wcols, cc = i - r * wcols;
      const int yy = by - kh + r, xx = bx - kh + cc;
      const float v = pw[i];
      pc[i] = (v != 0.0f) ? v * field_point(a.F, c, xx, yy) : 0.0f;
    }
    __syncthreads();
    // x correlation: xb[r][lx] = sum_j g_nx[j] pc[r][lx + j] (offset u = j - kh).
    const float* g = a.gx + o.x * ks;
    for (int it = tid; it < nrows * kGTW; it += blockDim.x) {
      const int r = it / kGTW, l = it - r * kGTW;
      const float* row = pc + r * wcols + l;
      float acc = 0.0f;
      for (int j = 0; j < ks; ++j) acc = fmaf(__ldg(g + j), row[j], acc);
      xb[r * kGTW + l] = acc;
    }
    __syncthreads();
    const float* gyy = a.gy + o.y * ks;
    for (int i = 0; i < kRows; ++i) {
      const int ly = ly0 + i * (kGThreads / kGTW);
      float acc = out[i];
      for (int j = 0; j < ks; ++j) acc = fmaf(__ldg(gyy + j), xb[(ly + j) * kGTW + lx], acc);
      out[i] = acc;
    }
  }
  for (int i = 0; i < kRows; ++i) {
    const int x = bx + lx, y = by + ly0 + i * (kGThreads / kGTW);
    if (x >= w || y >= h) continue;
    const size_t idx = static_cast<size_t>(y) * w + x;
    const float rv = __ldg(a.ref + idx);
    const bool replaced = (a.rmask && __ldg(a.rmask + idx) != 0) || !isfinite(rv);
    a.out[idx] = replaced ? 0.0f : out[i];
  }
}

// The reference adjoint for up to 40 taps (KSP = 8 KB, zero padded): grouped by
// nx, sum_ny first. Both correlations are linear, so
//   dchi2/dR = sum_nx g_nx (*)_x [ sum_ny g_ny (*)_y (p a_{nx,ny}) ]
// needs one x correlation per nx instead of one per component. A CTA of 256
// threads takes 128 window columns (a pair per lane, packed FMAs) by 32 output
// rows, 8 rows per thread; a_c p is blended into one window buffer while the
// other is read, the y sums stay in registers over the group's components, and
// the x correlation reads them from shared memory, one row per lane. FP32 FMA
// bound: about 1200 FMA per pixel at 28 components of 23 taps (0.14 ms for
// 2048^2 at 37.2 TFMA/s); one x and one y correlation per component with a
// scalar load per tap took 2.70 ms, this 0.44 ms.
constexpr int kArCols = 128;           // window columns of a tile
constexpr int kArRows = 32;            // output rows of a tile
constexpr int kArLdI = kArCols + 4;    // y sums: conflict-free 16-byte reads, a row per lane

template <int KB>
__global__ void __launch_bounds__(256, 2) k_adjoint_f(AdjRefArgs a, int n_max) {
  constexpr int KSP = 8 * KB, TW = kArCols - KSP, WR = kArRows + KSP;  // output columns, window rows
  extern __shared__ __align__(16) float smem[];
  float* pw = smem;                    // WR x kArCols: p
  float* pc = pw + WR * kArCols;       // 2 x WR x kArCols: p a_c
  float* ys = pc + 2 * WR * kArCols;   // kArRows x kArLdI: sum_ny g_ny (*)_y (p a_c)
  float* gx = ys + kArRows * kArLdI;   // (n_max + 1) x KSP
  float* gy = gx + (n_max + 1) * KSP;
  const int ks = a.ks, kh = (ks - 1) / 2, w = a.w, h = a.h, tid = threadIdx.x;
  const DevFields& F = a.F;
  const int bx = blockIdx.x * TW, by = blockIdx.y * kArRows;
  for (int i = tid; i < (n_max + 1) * KSP; i += 256) {
    const int q = i / KSP, j = i - q * KSP;
    gx[i] = j < ks ? a.gx[q * ks + j] : 0.0f;
    gy[i] = j < ks ? a.gy[q * ks + j] : 0.0f;
  }
  for (int i = tid; i < WR * kArCols; i += 256) {
    const int r = i / kArCols, c = i - r * kArCols;
    const int yy = by - kh + r, xx = bx - kh + c;
    pw[i] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? a.p[static_cast<size_t>(yy) * w + xx] : 0.0f;
  }
  // This thread's window columns (a pair) and rows: WR / 4 in the blend, 8 in the y correlation.
  const int cp = 2 * (tid & 63), rg = tid >> 6;
  int xc[2], jx[2];
  float wx[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    xc[u] = min(max(bx - kh + cp + u, 0), w - 1);
    jx[u] = F.exact ? 0 : F.cellx[xc[u]];
    wx[u] = F.exact ? 0.0f : F.wx[xc[u]];
  }
  auto blend = [&](int c, float* dst) {
    int cj = -1;
    float a00[2], e[2], t[2], g[2];
    for (int r = rg * (WR / 4); r < (rg + 1) * (WR / 4); ++r) {
      const int yy = min(max(by - kh + r, 0), h - 1);
      const float2 pv = *reinterpret_cast<const float2*>(pw + r * kArCols + cp);
      float f[2];
      if (F.exact) {
#pragma unroll
        for (int u = 0; u < 2; ++u) f[u] = __ldg(F.full + (static_cast<size_t>(c) * h + yy) * w + xc[u]);
      } else {
        const int jy = F.celly[yy];
        const float fy = F.wy[yy];
        if (jy != cj) {
          cj = jy;
          const float* r0 = F.latf + (static_cast<size_t>(c) * F.ncy + cj) * F.ncx;
          const float* r1 = r0 + F.ncx;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float b00 = __ldg(r0 + jx[u]), b01 = __ldg(r0 + jx[u] + 1);
            const float b10 = __ldg(r1 + jx[u]), b11 = __ldg(r1 + jx[u] + 1);
            a00[u] = b00;
            e[u] = b10 - b00;
            t[u] = b01 - b00;
            g[u] = (b11 - b10) - t[u];
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          f[u] = __fmaf_rn(__fmaf_rn(g[u], fy, t[u]), wx[u], __fmaf_rn(e[u], fy, a00[u]));
      }
      *reinterpret_cast<float2*>(dst + r * kArCols + cp) = make_float2(pv.x * f[0], pv.y * f[1]);
    }
  };
  // x correlation items: lane = row, 8 output columns per warp and step.
  constexpr int kGroups = TW / 8, kItems = (kGroups + 7) / 8;
  const int lane = tid & 31, warp = tid >> 5;
  float out[kItems][8];
#pragma unroll
  for (int n = 0; n < kItems; ++n)
#pragma unroll
    for (int i = 0; i < 8; ++i) out[n][i] = 0.0f;
  auto comp = [](int nx, int ny) { return (nx + ny) * (nx + ny + 1) / 2 + ny; };
  __syncthreads();
  blend(comp(0, 0), pc);
  int buf = 0;
  for (int nx = 0; nx <= n_max; ++nx) {
    float2 acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = make_float2(0.0f, 0.0f);
    for (int ny = 0; ny <= n_max - nx; ++ny) {
      __syncthreads();  // this component's window is complete, the other buffer is read
      const float* cur = pc + buf * WR * kArCols;
      buf ^= 1;
      if (ny < n_max - nx)
        blend(comp(nx, ny + 1), pc + buf * WR * kArCols);
      else if (nx < n_max)
        blend(comp(nx + 1, 0), pc + buf * WR * kArCols);
      const float* col = cur + rg * 8 * kArCols + cp;
      const float* g = gy + ny * KSP;
#pragma unroll
      for (int j0 = 0; j0 < KSP; j0 += 8) {
        const int nt = j0 + 8 < KSP ? 8 : a.ks - j0;  // taps of this block (the last: the rest are zeros)
        float2 v[15];
#pragma unroll
        for (int t = 0; t < 15; ++t)
          if (t < 7 + nt) v[t] = *reinterpret_cast<const float2*>(col + (j0 + t) * kArCols);
        const float4 ka = *reinterpret_cast<const float4*>(g + j0), kb = *reinterpret_cast<const float4*>(g + j0 + 4);
        const float kv[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          if (jj >= nt) break;
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = __ffma2_rn(make_float2(kv[jj], kv[jj]), v[i + jj], acc[i]);
        }
      }
    }
    // (the x pass of the previous nx finished reading ys before this nx's first barrier)
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<float2*>(ys + (rg * 8 + i) * kArLdI + cp) = acc[i];
    __syncthreads();
#pragma unroll
    for (int n = 0; n < kItems; ++n) {
      const int grp = warp + 8 * n;
      if (grp >= kGroups) break;
      const float* row = ys + lane * kArLdI + 8 * grp;
#pragma unroll
      for (int j0 = 0; j0 < KSP; j0 += 8) {
        float v[16];
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
          const float4 q = *reinterpret_cast<const float4*>(row + j0 + t);
          v[t] = q.x, v[t + 1] = q.y, v[t + 2] = q.z, v[t + 3] = q.w;
        }
        const float4 ka = *reinterpret_cast<const float4*>(gx + nx * KSP + j0);
        const float4 kb = *reinterpret_cast<const float4*>(gx + nx * KSP + j0 + 4);
        const float kv[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
        const int nt = j0 + 8 < KSP ? 8 : a.ks - j0;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          if (jj >= nt) break;
#pragma unroll
          for (int i = 0; i < 8; ++i) out[n][i] = __fmaf_rn(kv[jj], v[i + jj], out[n][i]);
        }
      }
    }
  }
  const int y = by + lane;
  if (y >= h) return;
#pragma unroll
  for (int n = 0; n < kItems; ++n) {
    const int grp = warp + 8 * n;
    if (grp >= kGroups) break;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int x = bx + 8 * grp + i;
      if (x >= w) break;
      const size_t idx = static_cast<size_t>(y) * w + x;
      const float rv = __ldg(a.ref + idx);
      const bool replaced = (a.rmask && __ldg(a.rmask + idx) != 0) || !isfinite(rv);
      a.out[idx] = replaced ? 0.0f : out[n][i];
    }
  }
}

template <int KB>
static void launch_adjoint_f(cudaStream_t st, const AdjRefArgs& a, int n_max) {
  constexpr int KSP = 8 * KB;
  const size_t smem = sizeof(float) * (3 * static_cast<size_t>(kArRows + KSP) * kArCols + kArRows * kArLdI +
                                       2 * static_cast<size_t>(n_max + 1) * KSP);
  auto kern = k_adjoint_f<KB>;
  ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
  kern<<<dim3(ceil_div(a.w, kArCols - KSP), ceil_div(a.h, kArRows)), 256, smem, st>>>(a, n_max);
  DGPU_LAUNCH("k_adjoint_f");
}

void launch_chi2_tile(cudaStream_t st, const Chi2Args& a, bool grad) {
  int blocks;
  if (launch_chi2_fast(st, a, grad, &blocks)) return;
  const dim3 grid(ceil_div(a.w, kGTW), ceil_div(a.h, kGTH));
  const size_t smem = chi2_tile_smem(a.n_max, a.ks);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_chi2_tile), smem);
  k_chi2_tile<<<grid, kGThreads, smem, st>>>(a);
  DGPU_LAUNCH("k_chi2_tile");
}

int chi2_tile_blocks(const Chi2Args& a, bool grad) {
  Chi2Args q = a;
  q.partial = nullptr;
  int blocks;
  return launch_chi2_fast(nullptr, q, grad, &blocks) ? blocks : ceil_div(a.w, kGTW) * ceil_div(a.h, kGTH);
}

void launch_sum_rows(cudaStream_t st, const double* part, int nrows, int ncols, double* out) {
  k_sum_rows<<<ncols, 256, 0, st>>>(part, nrows, ncols, out);
  DGPU_LAUNCH("k_sum_rows");
}

int theta_grad_blocks() { return 148 * 2; }

void launch_theta_grad(cudaStream_t st, int w, int h, int nf, int k, const float* q, const float* p, const DevFields& D,
                       double* part) {
  if (nf * k > 64 * 64) fail(DGPU_ERR_INVALID, "gradient: too many field coefficients");
  auto go = [&](auto kern, int nt) {
    const size_t smem = std::max(sizeof(float) * kTgWarps * (66 + 8 * nt) * kTgLd, sizeof(double) * kTgWarps * 32 * 8 * nt);
    ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    kern<<<dim3(theta_grad_blocks(), ceil_div(k, 8 * nt), ceil_div(nf, 32)), kTgWarps * 32, smem, st>>>(w, h, nf, k, q, p,
                                                                                                  D, part);
  };
  if (k <= 16)
    go(k_theta_grad<2>, 2);
  else
    go(k_theta_grad<4>, 4);
  DGPU_LAUNCH("k_theta_grad");
}

void launch_adjoint_reference(cudaStream_t st, const AdjRefArgs& a, int n_max) {
  switch ((a.ks + 7) / 8) {
    case 1: return launch_adjoint_f<1>(st, a, n_max);
    case 2: return launch_adjoint_f<2>(st, a, n_max);
    case 3: return launch_adjoint_f<3>(st, a, n_max);
    case 4: return launch_adjoint_f<4>(st, a, n_max);
    case 5: return launch_adjoint_f<5>(st, a, n_max);
    default: break;  // longer taps: the generic kernel
  }
  const dim3 grid(ceil_div(a.w, kGTW), ceil_div(a.h, kGTH));
  const size_t smem = adjoint_ref_smem(a.ks);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_adjoint_reference), smem);
  k_adjoint_reference<<<grid, kGThreads, smem, st>>>(a);
  DGPU_LAUNCH("k_adjoint_reference");
}

}  // namespace dgpu
