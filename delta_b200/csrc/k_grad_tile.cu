// chi^2 tiles of the kernel model (see k_grad.cu) for the common basis shapes:
// NX = n_max + 1 components per direction and the taps padded with zeros to
// KSP = 8 KB, both known at compile time. The x pass takes its taps in pairs: the one
// after the last is a zero, which times a finite staged value adds an exact zero. The y
// pass stops at the last tap. Every sum keeps the generic kernel's order (x taps, y taps
// and components ascending), so the per-pixel values are its values bit for bit.
//
// Value only (GRAD false): C_c alone. x sums as one float per column, y pass
// with 2 columns x 4 rows per thread in packed FMAs, 32 x 64 tiles, two CTAs
// per SM. Neither the derivative sums nor any per-pixel plane is formed:
// 2048^2, 28 components of 23 taps: 1.78 ms with the generic kernel (which
// always forms them), 0.29 ms now.
//
// With gradients: C, C^x and C^y per component. The x sums of g and g' lie side
// by side as one float2 per column, so one 8-byte load feeds the packed FMA
// (C, C^x) += g_y (t, t') and the scalar C^y += g'_y t; a thread holds 1 column
// x 8 rows, whose sliding window makes 15 loads serve 192 FMAs (with 4 rows the
// loads would bound it). The two buffers take 154 KB at 32 x 64, so one CTA of
// 256 threads per SM: 1.78 ms with the generic kernel, 0.81 ms now. FP32 FMA
// bound: 2500 FMA per pixel with the halo rows, 0.28 ms at 37.2 TFMA/s.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "grad_internal.h"

namespace dgpu {

namespace {

constexpr int kTW = 32;       // tile columns
constexpr int kPadCols = 8;   // zero columns left of the reference window
constexpr int kThreads = 256;

__host__ __device__ constexpr int window_cols(int ks) { return (kPadCols + kTW + (ks - 1) + 3) & ~3; }

template <int NX, int KB, bool GRAD>
struct Layout {
  static constexpr int KSP = 8 * KB;
  static constexpr int V = GRAD ? 2 : 1;  // floats per column of the x sums
  // Floats: reference window in row pairs, x sums, y taps (g_y, and g'_y), x
  // taps duplicated as (k, k) (g_x, and g'_x), lattice corners.
  static size_t floats(int TH, int ks, int lat) {
    const int nrows = TH + ks - 1;
    return 2 * static_cast<size_t>((nrows + 1) / 2) * window_cols(ks) +
           static_cast<size_t>(NX) * nrows * kTW * V + static_cast<size_t>(NX) * KSP * 3 * V + lat;
  }
};

// Floats for the lattice corners a tile of TH rows touches.
int lattice_floats(const DevFields& F, int TH) {
  if (F.exact || F.stride <= 0) return 0;
  const int lx = std::min(F.ncx, (kTW - 1) / F.stride + 3), ly = std::min(F.ncy, (TH - 1) / F.stride + 3);
  return F.nf * lx * ly;
}

template <int NX, int KB, bool GRAD>
__global__ void __launch_bounds__(kThreads, GRAD ? 1 : 2) k_chi2_f(Chi2Args a, int TH, int lat_cap) {
  using L = Layout<NX, KB, GRAD>;
  constexpr int KSP = L::KSP, V = L::V;
  extern __shared__ __align__(16) float smem[];
  const int ks = a.ks, kh = (ks - 1) / 2, w = a.w, h = a.h, nc = a.nc;
  const int nrows = TH + 2 * kh, wcols = kTW + 2 * kh, rw = window_cols(ks);
  const int npair = (nrows + 1) / 2;
  float* win = smem;                         // npair x rw row pairs; column kPadCols + c <-> frame column bx - kh + c
  float* tx = win + 2 * npair * rw;          // NX x nrows x kTW x V
  float* gy = tx + NX * nrows * kTW * V;     // NX x KSP, then (GRAD) g'_y
  float* gx2 = gy + NX * KSP * V;            // NX x KSP pairs, then (GRAD) g'_x
  float* slat = gx2 + 2 * NX * KSP * V;      // nf x lly x llx
  const int bx = blockIdx.x * kTW, by = blockIdx.y * TH, tid = threadIdx.x;
  const DevFields& F = a.F;
  const float fill = *a.fill;

  int lcx0 = 0, lcy0 = 0, llx = 0, lly = 0;
  bool staged = false;
  if (!F.exact) {
    lcx0 = F.cellx[bx];
    lcy0 = F.celly[by];
    llx = F.cellx[min(bx + kTW - 1, w - 1)] + 2 - lcx0;
    lly = F.celly[min(by + TH - 1, h - 1)] + 2 - lcy0;
    staged = F.nf * llx * lly <= lat_cap;
    if (staged)
      for (int i = tid; i < F.nf * lly * llx; i += kThreads) {
        const int f = i / (lly * llx), r = (i / llx) % lly, c = i % llx;
        slat[i] = __ldg(F.latf + (static_cast<size_t>(f) * F.ncy + lcy0 + r) * F.ncx + lcx0 + c);
      }
  }
  for (int i = tid; i < NX * KSP; i += kThreads) {
    const int q = i / KSP, j = i - q * KSP;
    const bool in = j < ks;
    gy[i] = in ? a.gy[q * ks + j] : 0.0f;
    reinterpret_cast<float2*>(gx2)[i] = in ? make_float2(a.gx[q * ks + j], a.gx[q * ks + j]) : make_float2(0.0f, 0.0f);
    if (GRAD) {
      gy[NX * KSP + i] = in ? a.dgy[q * ks + j] : 0.0f;
      reinterpret_cast<float2*>(gx2)[NX * KSP + i] =
          in ? make_float2(a.dgx[q * ks + j], a.dgx[q * ks + j]) : make_float2(0.0f, 0.0f);
    }
  }
  for (int i = tid; i < 2 * npair * rw; i += kThreads) {
    const int r = i / rw, cc = i - r * rw, c = cc - kPadCols;
    const int yy = by - kh + r, xx = bx - kh + c;
    float v = 0.0f;
    if (r < nrows && c >= 0 && c < wcols && yy >= 0 && yy < h && xx >= 0 && xx < w) {
      const size_t idx = static_cast<size_t>(yy) * w + xx;
      v = __ldg(a.ref + idx);
      if ((a.rmask && __ldg(a.rmask + idx) != 0) || !isfinite(v)) v = fill;
    }
    win[((r >> 1) * rw + cc) * 2 + (r & 1)] = v;
  }
  __syncthreads();

  // x pass: 2 columns x 2 rows x NX sums (x 2 tap sets) per thread, the row pair packed.
  for (int it = tid; it < npair * (kTW / 2); it += kThreads) {
    const int rp = it / (kTW / 2), c0 = 2 * (it - rp * (kTW / 2));
    const float2* row = reinterpret_cast<const float2*>(win) + rp * rw + kPadCols + c0 + 2 * kh;
    float2 acc[V][NX][2];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int q = 0; q < NX; ++q) acc[v][q][0] = acc[v][q][1] = make_float2(0.0f, 0.0f);
    float2 s0 = row[0], s1 = row[1];
#pragma unroll
    for (int j0 = 0; j0 < KSP; j0 += 2) {
      if (j0 > KSP - 8 && j0 >= ks) break;  // zero taps: the same for every thread
      float2 p0 = s0, p1 = s1;
      if (j0 > 0) {
        p1 = s0;
        p0 = row[-j0];
      }
      const float2 n0 = row[-j0 - 1];
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int q = 0; q < NX; ++q) {
          const float4 k = *reinterpret_cast<const float4*>(gx2 + 2 * ((v * NX + q) * KSP + j0));
          const float2 ka = make_float2(k.x, k.y), kb = make_float2(k.z, k.w);
          acc[v][q][0] = __ffma2_rn(kb, n0, __ffma2_rn(ka, p0, acc[v][q][0]));
          acc[v][q][1] = __ffma2_rn(kb, p0, __ffma2_rn(ka, p1, acc[v][q][1]));
        }
      s0 = n0;
    }
    const int r = 2 * rp;
#pragma unroll
    for (int q = 0; q < NX; ++q) {
      float* o = tx + ((q * nrows + r) * kTW + c0) * V;
      if (GRAD) {
        *reinterpret_cast<float4*>(o) = make_float4(acc[0][q][0].x, acc[V - 1][q][0].x, acc[0][q][1].x, acc[V - 1][q][1].x);
        if (r + 1 < nrows)
          *reinterpret_cast<float4*>(o + kTW * V) =
              make_float4(acc[0][q][0].y, acc[V - 1][q][0].y, acc[0][q][1].y, acc[V - 1][q][1].y);
      } else {
        *reinterpret_cast<float2*>(o) = make_float2(acc[0][q][0].x, acc[0][q][1].x);
        if (r + 1 < nrows) *reinterpret_cast<float2*>(o + kTW) = make_float2(acc[0][q][0].y, acc[0][q][1].y);
      }
    }
  }
  __syncthreads();

  constexpr int R = GRAD ? 8 : 4, COLS = GRAD ? 1 : 2;
  const int lx = COLS * (tid % (kTW / COLS)), ly = (tid / (kTW / COLS)) * R;
  const bool mine = ly < TH && bx + lx < w;
  double sums[4] = {0.0, 0.0, 0.0, 0.0};  // chi2, d/ds, d/ddx, d/ddy
  if (mine) {
    // a_f(x, y) of row i, column u: the lattice corners are re-read only when
    // the coarse cell row changes (cell_blend's operations and rounding).
    int jx[COLS], xc[COLS], jy[R];
    float wx[COLS], fy[R];
#pragma unroll
    for (int u = 0; u < COLS; ++u) {
      xc[u] = min(bx + lx + u, w - 1);
      jx[u] = F.exact ? 0 : F.cellx[xc[u]];
      wx[u] = F.exact ? 0.0f : F.wx[xc[u]];
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int y = min(by + ly + i, h - 1);
      jy[i] = F.exact ? 0 : F.celly[y];
      fy[i] = F.exact ? 0.0f : F.wy[y];
    }
    auto fields_of = [&](int f, float (&o)[R][COLS]) {
      if (F.exact) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int u = 0; u < COLS; ++u)
            o[i][u] = __ldg(F.full + (static_cast<size_t>(f) * h + min(by + ly + i, h - 1)) * w + xc[u]);
        return;
      }
      int cj = -1;
      float a00[COLS], e[COLS], t[COLS], g[COLS];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (jy[i] != cj) {
          cj = jy[i];
          const float* r0 = staged ? slat + (f * lly + (cj - lcy0)) * llx - lcx0
                                   : F.latf + (static_cast<size_t>(f) * F.ncy + cj) * F.ncx;
          const float* r1 = r0 + (staged ? llx : F.ncx);
#pragma unroll
          for (int u = 0; u < COLS; ++u) {
            const float b00 = r0[jx[u]], b01 = r0[jx[u] + 1], b10 = r1[jx[u]], b11 = r1[jx[u] + 1];
            a00[u] = b00;
            e[u] = b10 - b00;
            t[u] = b01 - b00;
            g[u] = (b11 - b10) - t[u];
          }
        }
#pragma unroll
        for (int u = 0; u < COLS; ++u)
          o[i][u] = __fmaf_rn(__fmaf_rn(g[u], fy[i], t[u]), wx[u], __fmaf_rn(e[u], fy[i], a00[u]));
      }
    };
    const size_t N = static_cast<size_t>(w) * h;
    const size_t at = static_cast<size_t>(by + ly) * w + bx + lx;
    float m0[R][COLS], mx[R][COLS], my[R][COLS];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int u = 0; u < COLS; ++u) m0[i][u] = mx[i][u] = my[i][u] = 0.0f;
    const int base = ly + 2 * kh;  // x-sum row of output row 0, tap 0
    for (int c = 0; c < nc; ++c) {
      const int2 o = a.orders[c];
      const float2* col = reinterpret_cast<const float2*>(tx + static_cast<size_t>(o.x) * nrows * kTW * V + lx * V);
      const float* g0 = gy + o.y * KSP;
      float2 cc[R];  // GRAD: (C, C^x) of row i; else C of the two columns
      float cy[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        cc[i] = make_float2(0.0f, 0.0f);
        cy[i] = 0.0f;
      }
#pragma unroll
      for (int j0 = 0; j0 < KSP; j0 += 8) {
        const int nt = j0 + 8 < KSP ? 8 : ks - j0;  // taps of this block (the last: the rest are zeros)
        float2 v[R + 7];                            // v[t] = x-sum row base - j0 - 7 + t
        const float2* vb = col + (base - j0 - 7) * (kTW * V / 2);
#pragma unroll
        for (int t = 0; t < R + 7; ++t)
          if (t >= 8 - nt) v[t] = vb[t * (kTW * V / 2)];
        const float4 ka = *reinterpret_cast<const float4*>(g0 + j0), kb = *reinterpret_cast<const float4*>(g0 + j0 + 4);
        const float kv[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
        float dv[8] = {};
        if (GRAD) {
          const float4 da = *reinterpret_cast<const float4*>(g0 + NX * KSP + j0);
          const float4 db = *reinterpret_cast<const float4*>(g0 + NX * KSP + j0 + 4);
          dv[0] = da.x, dv[1] = da.y, dv[2] = da.z, dv[3] = da.w;
          dv[4] = db.x, dv[5] = db.y, dv[6] = db.z, dv[7] = db.w;
        }
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          if (jj >= nt) break;
#pragma unroll
          for (int i = 0; i < R; ++i) {
            cc[i] = __ffma2_rn(make_float2(kv[jj], kv[jj]), v[i - jj + 7], cc[i]);
            if (GRAD) cy[i] = __fmaf_rn(dv[jj], v[i - jj + 7].x, cy[i]);
          }
        }
      }
      float f[R][COLS];
      fields_of(c, f);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        m0[i][0] = __fmaf_rn(f[i][0], cc[i].x, m0[i][0]);
        if (GRAD) {
          mx[i][0] = __fmaf_rn(f[i][0], cc[i].y, mx[i][0]);
          my[i][0] = __fmaf_rn(f[i][0], cy[i], my[i][0]);
          if (a.q && by + ly + i < h) a.q[static_cast<size_t>(c) * N + at + static_cast<size_t>(i) * w] = cc[i].x;
        } else {
          m0[i][COLS - 1] = __fmaf_rn(f[i][COLS - 1], cc[i].y, m0[i][COLS - 1]);
        }
      }
    }
    float bg[R][COLS];
    fields_of(nc, bg);
    const float s = a.scale;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int u = 0; u < COLS; ++u) {
        if (by + ly + i >= h || bx + lx + u >= w) continue;
        const size_t idx = at + static_cast<size_t>(i) * w + u;
        const float model = __fmaf_rn(s, m0[i][u], bg[i][u]);
        const float sv = __ldg(a.sci + idx), wt = __ldg(a.weight + idx);
        const bool ok = wt > 0.0f && isfinite(sv) && isfinite(model);
        const float r = ok ? sv - model : 0.0f;
        const float rb = ok ? -2.0f * wt * r : 0.0f;
        if (ok) {
          sums[0] += static_cast<double>(wt) * static_cast<double>(r) * static_cast<double>(r);
          if (GRAD) {
            sums[1] += static_cast<double>(rb) * static_cast<double>(m0[i][u]);
            sums[2] -= static_cast<double>(rb) * static_cast<double>(s) * static_cast<double>(mx[i][u]);
            sums[3] -= static_cast<double>(rb) * static_cast<double>(s) * static_cast<double>(my[i][u]);
          }
        }
        if (GRAD) {
          if (a.q) a.q[static_cast<size_t>(nc) * N + idx] = rb;
          if (a.p) a.p[idx] = rb * s;
        }
      }
  }
  // Fixed-order block reduction.
  __shared__ double red[4][kThreads / 32];
  constexpr int NS = GRAD ? 4 : 1;
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    double v = sums[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[k][tid >> 5] = v;
  }
  __syncthreads();
  if (tid < 4) {
    double t = 0.0;
    if (tid < NS)
      for (int i = 0; i < kThreads / 32; ++i) t += red[tid][i];
    a.partial[static_cast<size_t>(blockIdx.y * gridDim.x + blockIdx.x) * 4 + tid] = t;
  }
}

// Tile height: with gradients the largest of 64, 48, 32, 16 rows whose x sums
// fit one CTA per SM; values: 64 rows (two CTAs per SM at the common shapes).
template <int NX, int KB, bool GRAD>
int tile_height(const Chi2Args& a) {
  for (int th = 64; th >= 16; th -= 16)
    if (sizeof(float) * Layout<NX, KB, GRAD>::floats(th, a.ks, lattice_floats(a.F, th)) <= (GRAD ? 220 : 112) * 1024)
      return th;
  return 0;
}

template <int NX, int KB, bool GRAD>
bool launch(cudaStream_t st, const Chi2Args& a, int* blocks) {
  const int th = tile_height<NX, KB, GRAD>(a);
  if (th == 0) return false;
  const dim3 grid(ceil_div(a.w, kTW), ceil_div(a.h, th));
  *blocks = static_cast<int>(grid.x * grid.y);
  if (a.partial == nullptr) return true;  // asked for the block count only
  const int lat = lattice_floats(a.F, th);
  const size_t smem = sizeof(float) * Layout<NX, KB, GRAD>::floats(th, a.ks, lat);
  auto kern = k_chi2_f<NX, KB, GRAD>;
  ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
  kern<<<grid, kThreads, smem, st>>>(a, th, lat);
  DGPU_LAUNCH("k_chi2_f");
  return true;
}

template <int NX, int KB>
bool launch_kind(cudaStream_t st, const Chi2Args& a, bool grad, int* blocks) {
  return grad ? launch<NX, KB, true>(st, a, blocks) : launch<NX, KB, false>(st, a, blocks);
}

template <int NX>
bool launch_nx(cudaStream_t st, const Chi2Args& a, bool grad, int* blocks) {
  switch ((a.ks + 7) / 8) {
    case 2: return launch_kind<NX, 2>(st, a, grad, blocks);
    case 3: return launch_kind<NX, 3>(st, a, grad, blocks);
    case 4: return launch_kind<NX, 4>(st, a, grad, blocks);
    case 5: return launch_kind<NX, 5>(st, a, grad, blocks);
    default: return false;
  }
}

}  // namespace

bool launch_chi2_fast(cudaStream_t st, const Chi2Args& a, bool grad, int* blocks) {
  switch (a.n_max + 1) {
    case 3: return launch_nx<3>(st, a, grad, blocks);
    case 4: return launch_nx<4>(st, a, grad, blocks);
    case 5: return launch_nx<5>(st, a, grad, blocks);
    case 6: return launch_nx<6>(st, a, grad, blocks);
    case 7: return launch_nx<7>(st, a, grad, blocks);
    default: return false;
  }
}

}  // namespace dgpu
