// Full-frame subtraction kernels (sm_100a, FP32 SIMT):
//   * thin-plate field lattice / exact fields (FP64),
//   * fused tile model convolve D = S - b - sum_n a_n (g_ny *_y (g_nx *_x R~)),
//   * block-effective variance K^2 (x) Var(R) + Var(S),
//   * mask growth (separable OR dilation in shared memory) and exact-bad fill,
//   * radix-select upper median of a stride-7 sample (fill values).
// Reference: src/subtract.cpp:20-966.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <cstdlib>
#include <cmath>

#include "dev_common.cuh"
#include "select_internal.h"

namespace dgpu {

// ---------------------------------------------------------------------------
// Thin-plate fields
// ---------------------------------------------------------------------------

__device__ __forceinline__ double tps_green_d(double r2) { return r2 <= 0.0 ? 0.0 : 0.5 * r2 * log(r2); }

// fields(p, f) = design(p) . theta[f*k:(f+1)*k], design = [sigma Z | 1 | u | v]
// (src/spatial.cpp:67-97, src/subtract.cpp:58-63), of 32 points by a CTA: lane =
// point, the warps share the knots, then the design's columns, then the fields (each
// sum whole and in order in one thread). put(f, value) takes this lane's point. A
// thread per point doing all of it, its design row in local memory, took 17 us for
// the lattice of a 256 x 320 frame and 37 us at 4096 x 4096, now 6 and 12.
constexpr int kFieldPoints = 32;
size_t fields_smem(int k) { return sizeof(double) * 2 * kFieldPoints * static_cast<size_t>(k); }
template <class Put>
__device__ __forceinline__ void eval_fields(const TpsDev& t, const double* __restrict__ theta, int nf, double x, double y,
                                            Put put) {
  extern __shared__ __align__(16) double fsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int k = t.k, nr = k - 3;
  double* s = fsm + lane;                     // k x 32
  double* d = s + kFieldPoints * k;           // k x 32
  const double ux = (x - t.cx) / t.scale, uy = (y - t.cy) / t.scale;
  for (int j = warp; j < k; j += warps) {
    const double dx = ux - __ldg(t.kn + 2 * j), dy = uy - __ldg(t.kn + 2 * j + 1);
    s[j * kFieldPoints] = tps_green_d(dx * dx + dy * dy);
  }
  __syncthreads();
  for (int m = warp; m < k; m += warps) {
    double v = m == nr ? 1.0 : m == nr + 1 ? ux : uy;
    if (m < nr) {
      v = 0.0;
#pragma unroll 5
      for (int j = 0; j < k; ++j) v = fma(s[j * kFieldPoints], __ldg(t.z + j * nr + m), v);
    }
    d[m * kFieldPoints] = v;
  }
  __syncthreads();
  for (int f = warp; f < nf; f += warps) {
    const double* th = theta + static_cast<size_t>(f) * k;
    double acc = 0.0;
#pragma unroll 5
    for (int m = 0; m < k; ++m) acc = fma(d[m * kFieldPoints], __ldg(th + m), acc);
    put(f, acc);
  }
}

__global__ void __launch_bounds__(256) k_lattice(TpsDev t, const double* __restrict__ theta, int nf,
                                                 const int* __restrict__ gx, const int* __restrict__ gy, int ncx,
                                                 int ncy, double* __restrict__ lat, float* __restrict__ latf) {
  const int i = blockIdx.x * kFieldPoints + (threadIdx.x & 31), n = ncx * ncy;
  const int at = min(i, n - 1), ix = at % ncx, iy = at / ncx;
  eval_fields(t, theta, nf, static_cast<double>(gx[ix]), static_cast<double>(gy[iy]), [&](int f, double v) {
    if (i >= n) return;
    const size_t o = (static_cast<size_t>(f) * ncy + iy) * ncx + ix;
    lat[o] = v;
    latf[o] = static_cast<float>(v);
  });
}

__global__ void __launch_bounds__(256) k_exact_fields(TpsDev t, const double* __restrict__ theta, int nf, int w, int h,
                                                      float* __restrict__ full) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kFieldPoints + (threadIdx.x & 31), n = static_cast<int64_t>(w) * h;
  const int64_t at = min(i, n - 1);
  eval_fields(t, theta, nf, static_cast<double>(at % w), static_cast<double>(at / w), [&](int f, double v) {
    if (i < n) full[static_cast<size_t>(f) * n + i] = static_cast<float>(v);
  });
}

void launch_lattice(cudaStream_t s, const TpsDev& t, const double* theta, int nf, const int* gx,
                    const int* gy, int ncx, int ncy, double* lat, float* latf) {
  const int n = ncx * ncy;
  const size_t smem = fields_smem(t.k);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_lattice), smem);
  k_lattice<<<ceil_div(n, kFieldPoints), 256, smem, s>>>(t, theta, nf, gx, gy, ncx, ncy, lat, latf);
  DGPU_LAUNCH("k_lattice");
}

void launch_exact_fields(cudaStream_t s, const TpsDev& t, const double* theta, int nf, int w, int h,
                         float* full) {
  const int64_t n = static_cast<int64_t>(w) * h;
  const size_t smem = fields_smem(t.k);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_exact_fields), smem);
  k_exact_fields<<<ceil_div(n, kFieldPoints), 256, smem, s>>>(t, theta, nf, w, h, full);
  DGPU_LAUNCH("k_exact_fields");
}

// ---------------------------------------------------------------------------
// Fused model convolve (src/subtract.cpp:466-639).
//
// One CTA per 32 x TH output tile. The sanitised reference window (tile + kh
// halo, masked / non-finite -> fill, off-frame -> 0) is staged in shared
// memory; the NX = n_max+1 shared x-passes are computed into shared memory for
// the tile rows plus the y halo (each thread: 4 columns x all nx, sliding a
// 4-wide register window so every staged value is loaded once per tap); the
// y-pass of every component then runs out of shared memory with each thread
// holding 4 output rows of 2 adjacent columns in registers as float2 (taps in
// blocks of 8, the 11 row pairs a block touches in registers, one packed FMA
// per tap and row), and a_n / b are blended from the coarse lattice in
// registers, the corners re-read only when the coarse cell row changes. Per output
// pixel the accumulation order is the reference's: x taps j = 0..ks-1, then
// components in basis order, each y tap j ascending, d -= a_n * bn (FMA).
// Off-frame rows of the x-pass buffer are exact zeros, which leaves every
// clipped y sum bit-identical to the reference's jmin/jmax loop.
// ---------------------------------------------------------------------------

constexpr int kMcTW = 32;   // tile width (columns)
constexpr int kMcPad = 8;   // zero rows in front of each x-pass buffer (y-pass reads reach row -7)
constexpr int kMcYR = 4;    // output rows per thread in the y pass (2 columns each)
constexpr int kMcXPT = 4;   // output columns per thread in the x pass

// Tap rows in shared memory are padded to a multiple of 8 floats (zeros), so
// both passes read them as 16-byte vectors (the y pass reads 8 taps at j0 + 0..7).
__host__ __device__ constexpr int mc_tap_stride(int ks) { return (ks + 7) & ~7; }

template <int NX, bool STACK>
__global__ void __launch_bounds__(256)
k_model_convolve(int w, int h, const float* __restrict__ sci, const float* __restrict__ ref,
                 const uint8_t* __restrict__ rmask, DevFields F, const float* __restrict__ taps,
                 const int2* __restrict__ orders, int ks, int nc, const float* __restrict__ fillp,
                 float* __restrict__ diff, int TH) {
  // STACK == true is delta::basis_convolve (src/convolve.cpp:90-113): the raw
  // image (no sanitising), every component's B_n written to diff[n*h*w + ...].
  extern __shared__ __align__(16) float smem[];
  const int kh = (ks - 1) / 2;
  const int nrows = TH + 2 * kh;
  const int gbw = kMcTW + 2 * kh;
  const int gbw_pad = (gbw + 3) & ~3;
  const int kts = mc_tap_stride(ks);
  const int trows = nrows + kMcPad;
  float* rtile = smem;                                       // nrows x gbw_pad
  float* txs = rtile + nrows * gbw_pad;                      // NX x (kMcPad zero rows + nrows) x kMcTW
  float* ktaps = txs + NX * trows * kMcTW;                   // NX x kts (zero padded, 16-byte aligned rows)
  const int bx = blockIdx.x * kMcTW, by = blockIdx.y * TH;
  const float fill = STACK ? 0.0f : *fillp;
  const int tid = threadIdx.x;

  for (int i = tid; i < NX * kts; i += blockDim.x) {
    const int q = i / kts, j = i - q * kts;
    ktaps[i] = j < ks ? taps[q * ks + j] : 0.0f;
  }
  for (int i = tid; i < NX * kMcPad * kMcTW; i += blockDim.x) {
    const int q = i / (kMcPad * kMcTW);
    txs[q * trows * kMcTW + (i - q * kMcPad * kMcTW)] = 0.0f;
  }
  for (int i = tid; i < nrows * gbw; i += blockDim.x) {
    const int r = i / gbw, c = i - r * gbw;
    const int gy = by - kh + r, gx = bx - kh + c;
    float v = 0.0f;
    if (gy >= 0 && gy < h && gx >= 0 && gx < w) {
      const size_t idx = static_cast<size_t>(gy) * w + gx;
      v = __ldg(ref + idx);
      if (!STACK) {
        const bool bad = (rmask && __ldg(rmask + idx) != 0) || !isfinite(v);
        if (bad) v = fill;
      }
    }
    rtile[r * gbw_pad + c] = v;
  }
  __syncthreads();

  // ---- x pass: txs[nx][r][lx] = sum_j k[nx][j] * R~[y][x + kh - j] ----
  const int ngrp = kMcTW / kMcXPT;
  for (int it = tid; it < nrows * ngrp; it += blockDim.x) {
    const int r = it / ngrp, cg = it - r * ngrp;
    const int gy = by - kh + r;
    const int c0 = cg * kMcXPT;
    float acc[NX][kMcXPT];
#pragma unroll
    for (int q = 0; q < NX; ++q)
#pragma unroll
      for (int i = 0; i < kMcXPT; ++i) acc[q][i] = 0.0f;
    if (gy >= 0 && gy < h) {
      const float* row = rtile + r * gbw_pad + c0 + 2 * kh;  // column of tap j=0, output 0
      float win[kMcXPT];
#pragma unroll
      for (int i = 0; i < kMcXPT; ++i) win[i] = row[i];
      // Taps in groups of 4, one 16-byte load per component per group.
      for (int j0 = 0; j0 < ks; j0 += 4) {
        float4 kq[NX];
#pragma unroll
        for (int q = 0; q < NX; ++q) kq[q] = *reinterpret_cast<const float4*>(ktaps + q * kts + j0);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int j = j0 + jj;
          if (j >= ks) break;
          if (j > 0) {
#pragma unroll
            for (int i = kMcXPT - 1; i > 0; --i) win[i] = win[i - 1];
            win[0] = row[-j];
          }
#pragma unroll
          for (int q = 0; q < NX; ++q) {
            const float kc = jj == 0 ? kq[q].x : jj == 1 ? kq[q].y : jj == 2 ? kq[q].z : kq[q].w;
#pragma unroll
            for (int i = 0; i < kMcXPT; ++i) acc[q][i] = __fmaf_rn(kc, win[i], acc[q][i]);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < NX; ++q) {
      float4 v = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
      *reinterpret_cast<float4*>(txs + (q * trows + kMcPad + r) * kMcTW + c0) = v;
    }
  }
  __syncthreads();

  // ---- y pass + field blend: 2 adjacent columns x 4 rows per thread ----
  // Column pairs move as float2 (one 8-byte shared load per buffer row) and
  // every tap is one packed FMA (__ffma2_rn: an IEEE fma per lane, so each
  // output is the same FMA chain as a scalar loop).
  const int lx0 = 2 * (tid % (kMcTW / 2));
  const int ly0 = (tid / (kMcTW / 2)) * kMcYR;
  if (ly0 >= TH) return;
  const int x0 = bx + lx0;
  bool xin[2];
  int xcl[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    xin[u] = x0 + u < w;
    xcl[u] = xin[u] ? x0 + u : w - 1;
  }
  float2 d2[kMcYR];
  int jx[2] = {0, 0};
  float wxv[2] = {0.0f, 0.0f};
  int jy[kMcYR];
  float fy[kMcYR];
  if (!STACK && !F.exact) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      jx[u] = F.cellx[xcl[u]];
      wxv[u] = F.wx[xcl[u]];
    }
  }
#pragma unroll
  for (int i = 0; i < kMcYR; ++i) {
    const int y = min(by + ly0 + i, h - 1);
    if (!STACK && !F.exact) {
      jy[i] = F.celly[y];
      fy[i] = F.wy[y];
    } else {
      jy[i] = 0;
      fy[i] = 0.0f;
    }
  }
  // Field values a_f(x, y_i) of both columns; the lattice corners are re-read
  // only when the coarse cell row changes.
  auto fields_of = [&](int f, float2 (&a)[kMcYR]) {
    if (F.exact) {
#pragma unroll
      for (int i = 0; i < kMcYR; ++i) {
        const int y = min(by + ly0 + i, h - 1);
        const float* fr = F.full + (static_cast<size_t>(f) * h + y) * w;
        a[i] = make_float2(__ldg(fr + xcl[0]), __ldg(fr + xcl[1]));
      }
      return;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int cj = -1;
      float a00 = 0.0f, a01 = 0.0f, a10 = 0.0f, a11 = 0.0f;
#pragma unroll
      for (int i = 0; i < kMcYR; ++i) {
        if (jy[i] != cj) {
          cj = jy[i];
          const float* c0 = F.latf + (static_cast<size_t>(f) * F.ncy + cj) * F.ncx + jx[u];
          const float* c1 = c0 + F.ncx;
          a00 = __ldg(c0);
          a01 = __ldg(c0 + 1);
          a10 = __ldg(c1);
          a11 = __ldg(c1 + 1);
        }
        const float v = cell_blend(a00, a01, a10, a11, fy[i], wxv[u]);
        if (u == 0) a[i].x = v; else a[i].y = v;
      }
    }
  };
  if (!STACK) {
    float2 bg[kMcYR];
    fields_of(nc, bg);
#pragma unroll
    for (int i = 0; i < kMcYR; ++i) {
      const int y = min(by + ly0 + i, h - 1);
      const float* sr = sci + static_cast<size_t>(y) * w;
      d2[i] = make_float2(__ldg(sr + xcl[0]) - bg[i].x, __ldg(sr + xcl[1]) - bg[i].y);
    }
  }
  for (int n = 0; n < nc; ++n) {
    const int2 o = orders[n];
    // Row kMcPad of the component's buffer is row 0; the pad rows above are
    // zeros, so the reads of rows -7..-1 (taps past the top of the frame) need
    // no test.
    const float2* col =
        reinterpret_cast<const float2*>(txs + (static_cast<size_t>(o.x) * trows + kMcPad) * kMcTW + lx0);
    const float* ky = ktaps + o.y * kts;
    // Output row ly0+i needs buffer row ly0 + i + 2kh - j. Taps go in blocks of
    // 8 with the rows of a block held in registers (static indices), each
    // output still summing its taps j = 0..ks-1 in order.
    const int base = ly0 + 2 * kh;
    float2 bn[kMcYR];
#pragma unroll
    for (int i = 0; i < kMcYR; ++i) bn[i] = make_float2(0.0f, 0.0f);
    for (int j0 = 0; j0 < ks; j0 += 8) {
      float2 v[kMcYR + 7];  // v[t] = buffer row base - j0 - 7 + t
      const float2* vb = col + (base - j0 - 7) * (kMcTW / 2);
#pragma unroll
      for (int t = 0; t < kMcYR + 7; ++t) v[t] = vb[t * (kMcTW / 2)];
      const float4 ka = *reinterpret_cast<const float4*>(ky + j0);
      const float4 kb = *reinterpret_cast<const float4*>(ky + j0 + 4);
      const float kv[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        if (j0 + jj < ks) {
          const float c = kv[jj];
          const float2 cc = make_float2(c, c);
#pragma unroll
          for (int i = 0; i < kMcYR; ++i) bn[i] = __ffma2_rn(cc, v[i - jj + 7], bn[i]);
        }
      }
    }
    if (STACK) {
#pragma unroll
      for (int i = 0; i < kMcYR; ++i) {
        const int y = by + ly0 + i;
        if (y >= h) continue;
        float* dr = diff + (static_cast<size_t>(n) * h + y) * w;
        if (xin[0]) dr[x0] = bn[i].x;
        if (xin[1]) dr[x0 + 1] = bn[i].y;
      }
      continue;
    }
    float2 a[kMcYR];
    fields_of(n, a);
#pragma unroll
    for (int i = 0; i < kMcYR; ++i) d2[i] = __ffma2_rn(make_float2(-a[i].x, -a[i].y), bn[i], d2[i]);
  }
  if constexpr (!STACK) {
#pragma unroll
    for (int i = 0; i < kMcYR; ++i) {
      const int y = by + ly0 + i;
      if (y >= h) continue;
      const size_t o = static_cast<size_t>(y) * w + x0;
      if (xin[0] && xin[1] && (o & 1) == 0) {
        *reinterpret_cast<float2*>(diff + o) = d2[i];
      } else {
        if (xin[0]) diff[o] = d2[i].x;
        if (xin[1]) diff[o + 1] = d2[i].y;
      }
    }
  }
}

template <int NX, bool STACK>
static void launch_mc(cudaStream_t s, const SubtractArgs& a, const int2* orders, int TH, size_t smem) {
  auto kern = k_model_convolve<NX, STACK>;
  ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
  dim3 grid(ceil_div(a.w, kMcTW), ceil_div(a.h, TH));
  const int threads = (kMcTW / 2) * (TH / kMcYR);
  kern<<<grid, threads, smem, s>>>(a.w, a.h, a.sci, a.ref, a.ref_mask, a.F, a.taps, orders, a.ks,
                                   a.nc, a.fill, a.diff, TH);
  DGPU_LAUNCH("k_model_convolve");
}

size_t model_convolve_smem(int nx, int ks, int TH) {
  const int kh = (ks - 1) / 2;
  const int nrows = TH + 2 * kh;
  const int gbw_pad = ((kMcTW + 2 * kh) + 3) & ~3;
  return sizeof(float) * (static_cast<size_t>(nrows) * gbw_pad +
                          static_cast<size_t>(nx) * (nrows + kMcPad) * kMcTW + static_cast<size_t>(nx) * mc_tap_stride(ks));
}

size_t model_convolve_fast_smem(int nx, int ks, int TH, const DevFields& F);
bool model_convolve_fast_available(int nx, int ks);
bool launch_model_convolve_fast(cudaStream_t s, const SubtractArgs& a, const int2* orders, int TH);

static void launch_mc_th(cudaStream_t s, const SubtractArgs& a, const int2* orders, bool stack, int TH) {
  const int nx = a.n_max + 1;
  // The common basis shapes run the compile-time-shaped kernel (same bits;
  // DELTA_MODEL_CONVOLVE_GENERIC=1 forces this generic one, a diagnostic the
  // tests use to compare the two).
  const char* generic = std::getenv("DELTA_MODEL_CONVOLVE_GENERIC");
  if (!stack && !(generic && generic[0] == '1') && launch_model_convolve_fast(s, a, orders, TH)) return;
  const size_t smem = model_convolve_smem(nx, a.ks, TH);
  switch (nx) {
    case 1: stack ? launch_mc<1, true>(s, a, orders, TH, smem) : launch_mc<1, false>(s, a, orders, TH, smem); break;
    case 2: stack ? launch_mc<2, true>(s, a, orders, TH, smem) : launch_mc<2, false>(s, a, orders, TH, smem); break;
    case 3: stack ? launch_mc<3, true>(s, a, orders, TH, smem) : launch_mc<3, false>(s, a, orders, TH, smem); break;
    case 4: stack ? launch_mc<4, true>(s, a, orders, TH, smem) : launch_mc<4, false>(s, a, orders, TH, smem); break;
    case 5: stack ? launch_mc<5, true>(s, a, orders, TH, smem) : launch_mc<5, false>(s, a, orders, TH, smem); break;
    case 6: stack ? launch_mc<6, true>(s, a, orders, TH, smem) : launch_mc<6, false>(s, a, orders, TH, smem); break;
    case 7: stack ? launch_mc<7, true>(s, a, orders, TH, smem) : launch_mc<7, false>(s, a, orders, TH, smem); break;
    case 8: stack ? launch_mc<8, true>(s, a, orders, TH, smem) : launch_mc<8, false>(s, a, orders, TH, smem); break;
    case 9: stack ? launch_mc<9, true>(s, a, orders, TH, smem) : launch_mc<9, false>(s, a, orders, TH, smem); break;
    case 10: stack ? launch_mc<10, true>(s, a, orders, TH, smem) : launch_mc<10, false>(s, a, orders, TH, smem); break;
    case 11: stack ? launch_mc<11, true>(s, a, orders, TH, smem) : launch_mc<11, false>(s, a, orders, TH, smem); break;
    default: fail(DGPU_ERR_INVALID, "subtract: n_max above 10 is not supported by the tile engine");
  }
}

// The tile height is autotuned per (components, kernel size, frame size class):
// each height gives the same bits (the per-pixel order of every sum is fixed),
// only the redundant x-pass halo and the CTAs per SM differ. The first
// candidate is the heuristic: the tallest tile that still lets two CTAs share
// an SM, otherwise the tallest that fits.
void launch_model_convolve_orders(cudaStream_t s, const SubtractArgs& a, const int2* orders, bool stack) {
  const int nx = a.n_max + 1;
  const bool fast = !stack && model_convolve_fast_available(nx, a.ks);
  auto smem_of = [&](int th) { return fast ? model_convolve_fast_smem(nx, a.ks, th, a.F) : model_convolve_smem(nx, a.ks, th); };
  const size_t kTwoPerSm = 112 * 1024, kMaxSmem = 200 * 1024;
  int TH = 64;
  while (TH > 8 && smem_of(TH) > kTwoPerSm) TH /= 2;
  if (smem_of(TH) > kTwoPerSm) {
    TH = 64;
    while (TH > 8 && smem_of(TH) > kMaxSmem) TH /= 2;
  }
  if (smem_of(TH) > kMaxSmem) fail(DGPU_ERR_INVALID, "subtract: kernel footprint too large for the tile engine");
  std::vector<int> cands{TH};
  for (int t : {64, 32, 16})
    if (t != TH && smem_of(t) <= kMaxSmem) cands.push_back(t);
  int size_class = 0;
  for (int64_t px = static_cast<int64_t>(a.w) * a.h; px > 1; px >>= 2) ++size_class;
  // DELTA_MODEL_CONVOLVE_TH forces one candidate (a diagnostic: the tests
  // check that every tile height gives the same bits).
  if (const char* f = std::getenv("DELTA_MODEL_CONVOLVE_TH")) {
    const int th = std::atoi(f);
    if (std::find(cands.begin(), cands.end(), th) != cands.end()) {
      launch_mc_th(s, a, orders, stack, th);
      return;
    }
  }
  const std::string key = std::string("model_convolve") + (stack ? "/stack" : fast ? "/fast" : "") + "/nx" +
                          std::to_string(nx) +
                          "/ks" + std::to_string(a.ks) + "/px4^" + std::to_string(size_class);
  autotune(s, key, cands, [&](int th) { launch_mc_th(s, a, orders, stack, th); });
}

// ---------------------------------------------------------------------------
// Variance propagation (src/subtract.cpp:641-824): per 64x64 block, K frozen at
// the block centre, squared and mirrored, footprint shrunk to the centred box
// holding (1 - 1e-4f) of sum K^2, flat-window shortcut Q * Var(R) when the
// window's (max - min) <= 1e-3f * max, otherwise the dense correlation in
// (ly, lx) tap order; then + Var(S).
// ---------------------------------------------------------------------------

// 4 x 4 adjacent outputs per thread. A window row is kept as four planes of every
// fourth column, so that the 16 threads of a row read consecutive words and each
// step along the taps takes one new window value; four taps of a row come with one
// 16-byte load. That is 8 loads for 64 multiply-adds, which leaves the FP32 pipe the
// bound of the taps; the squares' ordered FP64 sums and the window come on top.
// 4096 x 4096: 166 us at radius 8, where columns 16 apart and taps one by one (8 loads
// for 16) took 211.

constexpr int kVarB = 64;
constexpr int kVarMaxRk = 64;
__host__ __device__ constexpr int var_tap_stride(int rk) { return (2 * rk + 1 + 3) & ~3; }
// Floats of a plane: room for the columns the padded taps reach, and odd, so that the
// two rows of outputs in a warp lie 16 banks apart.
__host__ __device__ constexpr int var_plane(int rk) { return ((kVarB + 2 * rk + 1 + 6) / 4) | 1; }

__global__ void __launch_bounds__(256)
k_variance(int w, int h, DevFields F, const float* __restrict__ phi, int rk, int nc,
           const float* __restrict__ var_s, const float* __restrict__ var_r,
           float* __restrict__ var_out) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ks = 2 * rk + 1;
  const int kk = ks * ks;
  // Window column c of a row lies at (c % 4) pw + c / 4.
  const int pw = var_plane(rk), rs = 4 * pw;
  float* k1 = reinterpret_cast<float*>(smraw);        // K (unsquared); then the taps, rows padded to whole fours
  float* win = k1 + ks * var_tap_stride(rk);          // (kVarB + 2 rk) rows
  float* kf = win + (kVarB + 2 * rk) * rs;            // kk, mirrored K^2
  float* an = kf + kk;                                // nc
  __shared__ double s_qsum;
  __shared__ double s_box[kVarMaxRk];
  __shared__ float s_min[8], s_max[8];
  const int tid = threadIdx.x;
  const int bx = blockIdx.x * kVarB, by = blockIdx.y * kVarB;
  const int bw = min(kVarB, w - bx), bh = min(kVarB, h - by);

  if (var_r != nullptr) {
    const int cpx = min(bx + bw / 2, w - 1), cpy = min(by + bh / 2, h - 1);
    for (int n = tid; n < nc; n += blockDim.x) an[n] = field_point(F, n, cpx, cpy);
    __syncthreads();
    // K at the block centre, squared, mirrored: kf[kk-1-i] = K[i]^2.
    for (int i = tid; i < kk; i += blockDim.x) {
      float k2 = 0.0f;
      for (int n = 0; n < nc; ++n) k2 = __fmaf_rn(an[n], __ldg(phi + static_cast<size_t>(n) * kk + i), k2);
      k1[i] = k2;
      kf[kk - 1 - i] = k2 * k2;
    }
    __syncthreads();
    // Warp 1, lane 0: qsum = sum_i double(K_i)^2 in index order (the squares
    // are exact in double). Warp 0: lane L sums the centred box of half-width
    // L (and L + 32) in row-major order. The other warps gather the window
    // meanwhile; every thread picks the first box reaching the target after
    // the barrier below.
    if (tid == 32) {
      double q = 0.0;
#pragma unroll 8
      for (int i = 0; i < kk; ++i) q = fma(static_cast<double>(k1[i]), static_cast<double>(k1[i]), q);
      s_qsum = q;
    } else if (tid < 32) {
      for (int hw = tid; hw < rk; hw += 32) {
        double box = 0.0;
        const int lo = rk - hw, hi = rk + hw;
        for (int yy = lo; yy <= hi; ++yy)
#pragma unroll 4
          for (int xx = lo; xx <= hi; ++xx) box += static_cast<double>(kf[yy * ks + xx]);
        s_box[hw] = box;
      }
    }
    // Gather the zero-padded window, its min / max and whether it is all finite.
    float lmin = INFINITY, lmax = -INFINITY;
    int finite = 1;
    const int iwh = bh + 2 * rk, iww = bw + 2 * rk;
    constexpr int kRows = 5;  // rows of a warp in flight together
    for (int r0 = tid >> 5; r0 < iwh; r0 += 8 * kRows)
      for (int c = tid & 31; c < rs; c += 32) {
        const int gx = bx - rk + c;
        const bool in = c < iww, xin = in && gx >= 0 && gx < w;
        float v[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          const int r = r0 + 8 * u, gy = by - rk + r;
          v[u] = (xin && r < iwh && gy >= 0 && gy < h) ? __ldg(var_r + static_cast<size_t>(gy) * w + gx) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          const int r = r0 + 8 * u;
          if (r >= iwh) break;
          win[r * rs + (c & 3) * pw + (c >> 2)] = v[u];
          if (in) {
            lmin = fminf(lmin, v[u]);
            lmax = fmaxf(lmax, v[u]);
            finite &= isfinite(v[u]) ? 1 : 0;
          }
        }
      }
    for (int o = 16; o > 0; o >>= 1) {
      lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
      lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    }
    if ((tid & 31) == 0) {
      s_min[tid >> 5] = lmin;
      s_max[tid >> 5] = lmax;
    }
    // A zero tap adds an exact +-0 to a sum that is never -0 when the window is
    // finite, so the reference's zero-tap skip only matters otherwise.
    const bool all_finite = __syncthreads_and(finite) != 0;
    float wmin = s_min[0], wmax = s_max[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) {
      wmin = fminf(wmin, s_min[i]);
      wmax = fmaxf(wmax, s_max[i]);
    }
    int hw = rk;
    {
      const double target = (1.0 - static_cast<double>(1e-4f)) * s_qsum;
      for (int b = 0; b < rk; ++b)
        if (s_box[b] >= target) {
          hw = b;
          break;
        }
    }
    const bool flat = wmax > 0.0f && (wmax - wmin) <= 1e-3f * wmax;
    const float q = static_cast<float>(s_qsum);
    const int lo = rk - hw, hi = rk + hw;
    // The taps of the box, rows padded with zeros (k1 is done with).
    const int nt = 2 * hw + 1, ts = (nt + 3) & ~3;
    for (int i = tid; i < nt * ts; i += blockDim.x) {
      const int r = i / ts, c = i - r * ts;
      k1[i] = c < nt ? kf[(lo + r) * ks + lo + c] : 0.0f;
    }
    __syncthreads();
    // Outputs: rows oy0 .. oy0 + 3, columns 4 tx .. 4 tx + 3. Per output the taps are
    // accumulated in (ly, lx) order.
    const int tx = tid & 15, oy0 = (tid >> 4) * 4;
    float acc[4][4] = {};
    if (flat) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = q * win[(oy0 + i + rk) * rs + ((rk + j) & 3) * pw + tx + ((rk + j) >> 2)];
    } else if (all_finite) {
      auto row = [&](int r, auto whole) {
        const float* wr = win + (oy0 + lo + r) * rs + tx;
        auto at = [&](int c) { return wr[(c & 3) * pw + (c >> 2)]; };  // window column 4 tx + c
        float v[7];
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = at(lo + k);
        auto taps = [&](int l, auto count) {
          constexpr int K = decltype(count)::value;
#pragma unroll
          for (int k = 3; k < 3 + K; ++k) v[k] = at(lo + l + k);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int ly = r - i;  // tap row
            if (!decltype(whole)::value && (ly < 0 || ly >= nt)) continue;
            const float4 c = *reinterpret_cast<const float4*>(k1 + ly * ts + l);
            const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(cv[k], v[k + j], acc[i][j]);
          }
        };
        int l = 0;
        for (; l + 4 <= nt; l += 4) {
          taps(l, std::integral_constant<int, 4>{});
#pragma unroll
          for (int k = 0; k < 3; ++k) v[k] = v[k + 4];
        }
        if (nt & 2)  // nt is odd
          taps(l, std::integral_constant<int, 3>{});
        else
          taps(l, std::integral_constant<int, 1>{});
      };
      for (int r = 0; r <= 2 * hw + 3; ++r) {
        if (r >= 3 && r < nt)
          row(r, std::true_type{});
        else
          row(r, std::false_type{});
      }
    } else {  // zero taps are skipped
      for (int r = 0; r <= 2 * hw + 3; ++r)
        for (int l = 0; l < nt; ++l)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int ly = r - i;
            if (ly < 0 || ly >= nt) continue;
            const float c = k1[ly * ts + l];
            if (c == 0.0f) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              acc[i][j] = fmaf(c, win[(oy0 + lo + r) * rs + ((lo + l + j) & 3) * pw + tx + ((lo + l + j) >> 2)], acc[i][j]);
          }
    }
    if (!flat)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f + acc[i][j];
    // Whole rows of four where every row starts on a 16-byte boundary.
    const bool vec = (w & 3) == 0 && ((reinterpret_cast<uintptr_t>(var_out) | reinterpret_cast<uintptr_t>(var_s)) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int oy = oy0 + i;
      if (oy >= bh) continue;
      const size_t o = static_cast<size_t>(by + oy) * w + bx + 4 * tx;
      if (vec && 4 * tx + 3 < bw) {
        float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (var_s) {
          const float4 sv = __ldg(reinterpret_cast<const float4*>(var_s + o));
          v = make_float4(v.x + sv.x, v.y + sv.y, v.z + sv.z, v.w + sv.w);
        }
        *reinterpret_cast<float4*>(var_out + o) = v;
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (4 * tx + j >= bw) continue;
        float v = acc[i][j];
        if (var_s) v = v + __ldg(var_s + o + j);
        var_out[o + j] = v;
      }
    }
  } else {
    for (int p = tid; p < bw * bh; p += blockDim.x) {
      const int oy = p / bw, ox = p - oy * bw;
      const size_t o = static_cast<size_t>(by + oy) * w + bx + ox;
      var_out[o] = 0.0f + __ldg(var_s + o);
    }
  }
}

void launch_variance(cudaStream_t s, int w, int h, const DevFields& F, const float* phi, int rk,
                     int nc, const float* var_s, const float* var_r, float* var_out) {
  const int ks = 2 * rk + 1;
  const int iw = kVarB + 2 * rk;
  // What is refused: more than 200 KB without the padding.
  if (sizeof(float) * (2 * static_cast<size_t>(ks) * ks + static_cast<size_t>(iw) * iw + nc + 4) > 200 * 1024 ||
      rk > kVarMaxRk)
    fail(DGPU_ERR_INVALID, "subtract: kernel radius too large for the variance engine");
  const size_t smem = sizeof(float) * (static_cast<size_t>(ks) * var_tap_stride(rk) + static_cast<size_t>(iw) * 4 * var_plane(rk) +
                                       static_cast<size_t>(ks) * ks + nc + 4);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_variance), smem);
  dim3 grid(ceil_div(w, kVarB), ceil_div(h, kVarB));
  k_variance<<<grid, 256, smem, s>>>(w, h, F, phi, rk, nc, var_s, var_r, var_out);
  DGPU_LAUNCH("k_variance");
}

// ---------------------------------------------------------------------------
// Mask growth (src/subtract.cpp:826-914): science-side flags 1:1, reference
// flags and saturated reference pixels OR-dilated by r (box), edge border r,
// non-finite difference. exact_bad records the undilated garbage pixels for the fill
// pass. One CTA per T x T tile, four pixels to a 32-bit word: the grow window's words
// are ORed along x from byte-shifted pairs (most are zero and skipped), then along y,
// where a thread's four rows share the rows common to them. A byte per pixel, 2 r + 1
// of them per output and direction, took 213 us at 4096 x 4096, radius 8, now 87.
// ---------------------------------------------------------------------------

template <int T>
__global__ void __launch_bounds__(T * T / 16)
k_mask(int w, int h, const float* __restrict__ sci, const float* __restrict__ ref,
       const uint8_t* __restrict__ sm, const uint8_t* __restrict__ rm, int has_sat, float sat, int r,
       const float* __restrict__ diff, uint8_t* __restrict__ mask_out, uint8_t* __restrict__ exact_bad, int vec) {
  extern __shared__ uint32_t msm32[];
  constexpr int TW = T / 4;                    // words of a tile row
  const int r4 = (r + 3) & ~3, gh = T + 2 * r, gw = (T + 2 * r4) / 4;
  uint32_t* g = msm32;          // gh x gw words: columns from bx - r4
  uint32_t* gxr = g + gh * gw;  // gh x TW after the x dilation
  const int bx = blockIdx.x * T, by = blockIdx.y * T;
  const int tid = threadIdx.x;
  // Flags that grow, of the four pixels from (x, y) on.
  auto grow_word = [&](int x, int y) {
    uint32_t v = 0;
    if (y < 0 || y >= h || x + 3 < 0 || x >= w) return v;
    const int64_t idx = static_cast<int64_t>(y) * w + x;
    if (vec && x >= 0 && x + 3 < w) {
      if (rm) v = __ldg(reinterpret_cast<const uint32_t*>(rm + idx));
      if (has_sat) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(ref + idx));
        v |= (f.x >= sat ? 0x2u : 0u) | (f.y >= sat ? 0x200u : 0u) | (f.z >= sat ? 0x20000u : 0u) |
             (f.w >= sat ? 0x2000000u : 0u);
      }
      return v;
    }
    for (int k = 0; k < 4; ++k) {
      if (x + k < 0 || x + k >= w) continue;
      uint32_t m = rm ? rm[idx + k] : 0u;
      if (has_sat && ref[idx + k] >= sat) m |= 2u;
      v |= m << (8 * k);
    }
    return v;
  };
  const bool need_grow = (rm != nullptr) || has_sat;
  if (need_grow) {
    for (int i = tid; i < gh * gw; i += blockDim.x) {
      const int yy = i / gw, xx = i - yy * gw;
      g[i] = grow_word(bx - r4 + 4 * xx, by - r + yy);
    }
    __syncthreads();
    for (int i = tid; i < gh * TW; i += blockDim.x) {
      const int yy = i / TW, o = i - yy * TW;
      const uint32_t* row = g + yy * gw + o;
      const int b0 = r4 - r, last = (b0 + 2 * r + 3) >> 2;  // first byte; last word of the window
      uint32_t any = 0;
      for (int k = 0; k <= last; ++k) any |= row[k];
      uint32_t acc = 0;
      if (any) {
        for (int d = b0; d <= b0 + 2 * r; ++d) {
          const int k = d >> 2;
          acc |= __funnelshift_r(row[k], k < last ? row[k + 1] : 0u, 8 * (d & 3));
        }
      }
      gxr[i] = acc;
    }
    __syncthreads();
  }
  const int o = tid % TW, ly0 = tid / TW * 4, x0 = bx + 4 * o;
  if (x0 >= w) return;
  uint32_t grown[4] = {0, 0, 0, 0};
  if (need_grow) {
    // Rows ly0 + i .. ly0 + i + 2 r; those from 3 to 2 r belong to all four.
    const uint32_t* col = gxr + ly0 * TW + o;
    if (2 * r >= 3) {
      uint32_t mid = 0;
      for (int d = 3; d <= 2 * r; ++d) mid |= col[d * TW];
      const uint32_t c0 = col[0], c1 = col[TW], c2 = col[2 * TW];
      const uint32_t e1 = col[(2 * r + 1) * TW], e2 = col[(2 * r + 2) * TW], e3 = col[(2 * r + 3) * TW];
      grown[0] = mid | c0 | c1 | c2;
      grown[1] = mid | c1 | c2 | e1;
      grown[2] = mid | c2 | e1 | e2;
      grown[3] = mid | e1 | e2 | e3;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        for (int d = 0; d <= 2 * r; ++d) grown[i] |= col[(i + d) * TW];
    }
  }
  const bool whole = vec && x0 + 3 < w;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int y = by + ly0 + i;
    if (y >= h) break;
    const size_t idx = static_cast<size_t>(y) * w + x0;
    uint32_t sw = 0, rw = 0;
    float rv[4] = {}, sv[4] = {}, dv[4] = {};
    const int n = min(4, w - x0);
    if (whole) {
      if (sm) sw = __ldg(reinterpret_cast<const uint32_t*>(sm + idx));
      if (rm) rw = __ldg(reinterpret_cast<const uint32_t*>(rm + idx));
      const float4 d = __ldg(reinterpret_cast<const float4*>(diff + idx));
      dv[0] = d.x, dv[1] = d.y, dv[2] = d.z, dv[3] = d.w;
      if (has_sat) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(ref + idx)), c = __ldg(reinterpret_cast<const float4*>(sci + idx));
        rv[0] = a.x, rv[1] = a.y, rv[2] = a.z, rv[3] = a.w;
        sv[0] = c.x, sv[1] = c.y, sv[2] = c.z, sv[3] = c.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k >= n) break;
        if (sm) sw |= static_cast<uint32_t>(sm[idx + k]) << (8 * k);
        if (rm) rw |= static_cast<uint32_t>(rm[idx + k]) << (8 * k);
        dv[k] = diff[idx + k];
        if (has_sat) {
          rv[k] = ref[idx + k];
          sv[k] = sci[idx + k];
        }
      }
    }
    uint32_t m = sw | grown[i], eb = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int x = x0 + k;
      uint32_t f = 0;
      bool bad = ((sw | rw) >> (8 * k) & 0xffu) != 0;
      if (has_sat) {
        if (rv[k] >= sat) bad = true;
        if (sv[k] >= sat) {
          f = 2;
          bad = true;
        }
      }
      if (x < r || x >= w - r || y < r || y >= h - r) f |= 16;
      if (!isfinite(dv[k])) {
        f |= 8;
        bad = true;
      }
      m |= f << (8 * k);
      eb |= (bad ? 1u : 0u) << (8 * k);
    }
    if (whole) {
      *reinterpret_cast<uint32_t*>(mask_out + idx) = m;
      *reinterpret_cast<uint32_t*>(exact_bad + idx) = eb;
    } else {
      for (int k = 0; k < n; ++k) {
        mask_out[idx + k] = static_cast<uint8_t>(m >> (8 * k));
        exact_bad[idx + k] = static_cast<uint8_t>(eb >> (8 * k));
      }
    }
  }
}

static size_t mask_smem(int t, int r) {
  return static_cast<size_t>(t + 2 * r) * (t + 2 * ((r + 3) & ~3) + t);
}

void launch_mask(cudaStream_t s, int w, int h, const float* sci, const float* ref,
                 const uint8_t* sm, const uint8_t* rm, double saturation, int r, const float* diff,
                 uint8_t* mask_out, uint8_t* exact_bad) {
  if (static_cast<size_t>(32 + 2 * r) * (64 + 2 * r) > 200 * 1024)
    fail(DGPU_ERR_INVALID, "subtract: kernel radius too large for mask growth");
  const int has_sat = saturation > 0.0 ? 1 : 0;
  const float sat = static_cast<float>(saturation);
  // Words of four pixels need rows that start on their boundaries.
  const uintptr_t bits = reinterpret_cast<uintptr_t>(sci) | reinterpret_cast<uintptr_t>(ref) | reinterpret_cast<uintptr_t>(diff);
  const uintptr_t bytes = reinterpret_cast<uintptr_t>(sm) | reinterpret_cast<uintptr_t>(rm) |
                          reinterpret_cast<uintptr_t>(mask_out) | reinterpret_cast<uintptr_t>(exact_bad);
  const int vec = (w & 3) == 0 && (bits & 15) == 0 && (bytes & 3) == 0;
  // Tiles of 64, whose windows overlap less, once there are two for every SM (below
  // that 32 x 32 ones fill more of them).
  auto go = [&](auto kern, int t) {
    const size_t smem = mask_smem(t, r);
    ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    kern<<<dim3(ceil_div(w, t), ceil_div(h, t)), t * t / 16, smem, s>>>(w, h, sci, ref, sm, rm, has_sat, sat, r, diff,
                                                                       mask_out, exact_bad, vec);
    DGPU_LAUNCH("k_mask");
  };
  if (static_cast<int64_t>(ceil_div(w, 64)) * ceil_div(h, 64) >= 2 * 148 && mask_smem(64, r) <= 100 * 1024)
    go(k_mask<64>, 64);
  else
    go(k_mask<32>, 32);
}

__global__ void k_mask_fill(int64_t n, const uint8_t* __restrict__ mask,
                            const uint8_t* __restrict__ exact_bad, const float* __restrict__ fillp,
                            float* __restrict__ diff, float* __restrict__ var) {
  const float fill = *fillp;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (mask[i] != 0 && exact_bad[i]) {
      diff[i] = fill;
      if (var) var[i] = 0.0f;
    }
  }
}

void launch_mask_fill(cudaStream_t s, int64_t n, const uint8_t* mask, const uint8_t* exact_bad,
                      const float* fill, float* diff, float* var) {
  const int blocks = static_cast<int>(std::min<int64_t>(ceil_div(n, 256), 148 * 16));
  k_mask_fill<<<blocks, 256, 0, s>>>(n, mask, exact_bad, fill, diff, var);
  DGPU_LAUNCH("k_mask_fill");
}

// Upper median of a stride-7 sample (std::nth_element(size / 2); an empty sample
// yields 0): the good finite reference pixels (src/subtract.cpp:20-51), or the
// unmasked finite difference pixels under the grown mask (915-945).
void launch_strided_median(Context& c, int64_t n, const float* values, const uint8_t* mask, float* d_result) {
  launch_upper_median(c, n, 7, values, mask, d_result);
}

// photometric_scale (src/fit.cpp:513-530): out = sum_c float(S_c) * a_c in
// component order, fused.
__global__ void k_photometric_scale(DevFields F, const float* __restrict__ sums, int nc,
                                    float* __restrict__ out) {
  const int64_t n = static_cast<int64_t>(F.w) * F.h;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int x = static_cast<int>(i % F.w), y = static_cast<int>(i / F.w);
    float acc = 0.0f;
    for (int q = 0; q < nc; ++q) acc = __fmaf_rn(sums[q], field_point(F, q, x, y), acc);
    out[i] = acc;
  }
}

void launch_photometric_scale(cudaStream_t s, const DevFields& F, const float* sums, int nc, float* out) {
  const int64_t n = static_cast<int64_t>(F.w) * F.h;
  const int blocks = static_cast<int>(std::min<int64_t>(ceil_div(n, 256), 148 * 16));
  k_photometric_scale<<<blocks, 256, 0, s>>>(F, sums, nc, out);
  DGPU_LAUNCH("k_photometric_scale");
}

// Transients-positive sign flip of the difference (python/delta/pipeline.py:687-689),
// in place: float4 body, scalar tail.
// v = v * scale (float32 product, the scalar rounded to float first), or
// v = value everywhere when fill is set.
__global__ void k_scale_fill(int64_t n, float* __restrict__ v, float scale, int fill, float value) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    v[i] = fill ? value : v[i] * scale;
}

void launch_scale_fill(cudaStream_t s, int64_t n, float* v, float scale, bool fill, float value) {
  const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 148 * 16));
  k_scale_fill<<<std::max(blocks, 1), 256, 0, s>>>(n, v, scale, fill ? 1 : 0, value);
  DGPU_LAUNCH("k_scale_fill");
}

__global__ void k_negate(int64_t n, float* __restrict__ v) {
  const int64_t n4 = (reinterpret_cast<uintptr_t>(v) & 15) ? 0 : n / 4;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  float4* v4 = reinterpret_cast<float4*>(v);
  for (int64_t i = t; i < n4; i += stride) {
    float4 a = v4[i];
    a.x = -a.x;
    a.y = -a.y;
    a.z = -a.z;
    a.w = -a.w;
    v4[i] = a;
  }
  for (int64_t i = 4 * n4 + t; i < n; i += stride) v[i] = -v[i];
}

void launch_negate(cudaStream_t s, int64_t n, float* v) {
  if (n <= 0) return;
  const int blocks = static_cast<int>(std::min<int64_t>(ceil_div(ceil_div(n, 4), 256), 148 * 8));
  k_negate<<<blocks, 256, 0, s>>>(n, v);
  DGPU_LAUNCH("k_negate");
}

// Device memory -> the context's mapped pinned read-back area by SM stores:
// range blockIdx.y of the list (16 bytes at a time when both ends are 16-byte
// aligned).
__global__ void k_read_back(ReadBackList l) {
  const int it = blockIdx.y;
  if (it >= l.n) return;
  const unsigned char* __restrict__ src = l.src[it];
  unsigned char* dst = l.dst[it];
  const size_t n = l.bytes[it];
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  size_t head = 0;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
    const size_t n16 = n / 16;
    for (size_t i = t; i < n16; i += stride)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    head = n16 * 16;
  }
  for (size_t i = head + t; i < n; i += stride) dst[i] = src[i];
}

void launch_read_back(cudaStream_t s, const ReadBackList& l) {
  if (l.n <= 0) return;
  unsigned long long most = 0;
  for (int i = 0; i < l.n; ++i) most = std::max(most, l.bytes[i]);
  const unsigned bx = static_cast<unsigned>(std::min<unsigned long long>((most + 4095) / 4096, 32));
  k_read_back<<<dim3(std::max(bx, 1u), static_cast<unsigned>(l.n)), 256, 0, s>>>(l);
  DGPU_LAUNCH("k_read_back");
}

}  // namespace dgpu

// ---------------------------------------------------------------------------
// Median of z^2 = D^2 / Var over the good pixels, exactly as numpy's median of
// the FP64 values (python/delta/pipeline.py's _variance_rescale_factor): the
// two middle ranks (lo = (m-1)/2, hi = m/2) of the FP64 keys found by one
// 64-bit radix select (8 passes of 8-bit digits, both ranks per pass), then
// (a + b) / 2 on the host. z^2 >= 0 and finite, so the keys order as their bit
// patterns. Good pixels: Var > 0, D and Var finite, mask 0.
// ---------------------------------------------------------------------------
namespace dgpu {

__global__ void k_z2_keys(int64_t n, const float* __restrict__ d, const float* __restrict__ v,
                          const uint8_t* __restrict__ m, unsigned long long* __restrict__ keys,
                          unsigned long long* __restrict__ count) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float dv = d[i], vv = v[i];
    if (!(vv > 0.0f) || !isfinite(dv) || !isfinite(vv) || (m && m[i] != 0)) continue;
    const double x = static_cast<double>(dv);
    const double z2 = x * x / static_cast<double>(vv);
    keys[atomicAdd(count, 1ull)] = static_cast<unsigned long long>(__double_as_longlong(z2));
  }
}

// state: [0] count, [1] rank lo, [2] rank hi, [3] prefix lo, [4] prefix hi; hist: 2 x 256.
__global__ void k_z2_hist(const unsigned long long* __restrict__ keys, unsigned long long* __restrict__ state,
                          int shift, unsigned int* __restrict__ hist) {
  __shared__ unsigned int h[2][256];
  for (int i = threadIdx.x; i < 512; i += blockDim.x) h[i >> 8][i & 255] = 0;
  __syncthreads();
  const unsigned long long n = state[0];
  const unsigned long long himask = shift >= 56 ? 0ull : (~0ull << (shift + 8));
  const unsigned long long p0 = state[3] & himask, p1 = state[4] & himask;
  for (unsigned long long i = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    const unsigned long long k = keys[i];
    const unsigned dgt = static_cast<unsigned>((k >> shift) & 0xffull);
    if ((k & himask) == p0) atomicAdd(&h[0][dgt], 1u);
    if ((k & himask) == p1) atomicAdd(&h[1][dgt], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const unsigned c = h[i >> 8][i & 255];
    if (c) atomicAdd(&hist[i], c);
  }
}

__global__ void k_z2_pick(unsigned long long* __restrict__ state, int shift, unsigned int* __restrict__ hist) {
  if (threadIdx.x >= 2) return;
  const int t = threadIdx.x;
  unsigned long long rank = state[1 + t];
  unsigned long long cum = 0;
  int d = 0;
  for (; d < 256; ++d) {
    const unsigned long long c = hist[t * 256 + d];
    if (rank < cum + c) break;
    cum += c;
  }
  if (d > 255) d = 255;  // unreachable while the rank is below the count
  state[1 + t] = rank - cum;
  state[3 + t] |= static_cast<unsigned long long>(d) << shift;
}

__global__ void k_z2_init(unsigned long long* __restrict__ state) {
  if (threadIdx.x == 0) {
    const unsigned long long n = state[0];
    state[1] = n ? (n - 1) / 2 : 0;
    state[2] = n / 2;
    state[3] = 0;
    state[4] = 0;
  }
}

void launch_z2_median(cudaStream_t s, int64_t n, const float* d, const float* v, const uint8_t* m,
                      unsigned long long* keys, unsigned long long* state, unsigned int* hist) {
  DGPU_CUDA(cudaMemsetAsync(state, 0, 5 * sizeof(unsigned long long), s));
  const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 148 * 8));
  k_z2_keys<<<std::max(blocks, 1), 256, 0, s>>>(n, d, v, m, keys, state);
  DGPU_LAUNCH("k_z2_keys");
  k_z2_init<<<1, 32, 0, s>>>(state);
  DGPU_LAUNCH("k_z2_init");
  for (int shift = 56; shift >= 0; shift -= 8) {
    DGPU_CUDA(cudaMemsetAsync(hist, 0, 512 * sizeof(unsigned int), s));
    k_z2_hist<<<std::max(blocks, 1), 256, 0, s>>>(keys, state, shift, hist);
    DGPU_LAUNCH("k_z2_hist");
    k_z2_pick<<<1, 32, 0, s>>>(state, shift, hist);
    DGPU_LAUNCH("k_z2_pick");
  }
}

}  // namespace dgpu
