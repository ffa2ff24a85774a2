// Panels of (ia|jb) for a block of occupied orbitals i0 <= i < i0 + ni and all
// j >= i0: the energy of the plain form from FP64-accurate panels
// (run_canonical_mp2_ri, src/POSTHF/can_mp2.cc:53-132), and the elementwise
// step of the adjoint.
//
// The panel is a product on the digit GEMM (dgemm_tc.cu): on this GPU an FP64
// fused multiply-add runs at two per clock per SM, 1.2 TFLOP/s, the digit GEMM
// at up to 53 TFLOP/s.  Its error is below the FP64 GEMM's relative to the norms
// of the rows (2e-16 to 7e-16 against 1.6e-15 to 3.5e-15 on integrals of real
// Gaussians, naux 192 to 1536) and a quarter to 2.2 times it relative to the
// elements' root mean square there; with the diagonal in FP64 the energy and the
// gradient are closer to extended precision than on the FP64 pipe.  Only j >= i0 is formed: (ia|jb) = (jb|ia).  The panel of a block (at most kPanelBudget)
// goes through HBM once: 16 bytes per element against 2 naux / 53e12 s, less
// than a tenth of the product from naux = 600 on.
#include <algorithm>

#include "common.cuh"
#include "dgemm_tc.h"
#include "fp64_approx.cuh"
#include "kernels.h"
#include "panel.h"

namespace corr {

namespace {

constexpr int PT = 32;  // tile edge

// CTAs of an (i, j) block of the panel (blockIdx.x) share its columns of 32 x 32
// tile pairs (A <= B, column B to blockIdx.y): with one CTA per block the 276
// blocks of 23 occupied orbitals left most of the GPU waiting for one another's
// loads (energy nocc=23 nvir=211: 187 us against 278 us).  A thread owns the pair (a, b), (b, a), the transposed tile comes (and goes back)
// through shared memory, so every access to the panel is coalesced.  Diagonal
// tiles see each pair from both sides at weight 1/2.
//
// GRAD = false: {E_OS, E_SS} of the pairs (i, j), (j, i) into the CTA's partial
// (j < i, which the block's own columns contain too, adds nothing).
// GRAD = true: every element becomes G_ab = -(4 M_ab - 2 M_ba) / D, and for
// j >= i W_ab = (2 M_ab - M_ba) M_ab / D^2 of both ordered pairs goes into
// dE/d eps, -sum (2 M_ab - M_ba) M_ab / D into the partial.
//
// Bound by the FP64 pipe: 10 (energy) or 16 (gradient) instructions per pair.
template <bool GRAD>
__global__ void __launch_bounds__(256) panel_kernel(PanelView pv, const double* __restrict__ eps,
                                                    double* __restrict__ deps,
                                                    double* __restrict__ part) {
  extern __shared__ double wv[];  // GRAD: [v] sums of W
  __shared__ double st[PT][PT + 1];
  __shared__ double red[2][8];
  const int o = pv.o, v = pv.v;
  const int nj = o - pv.i0;
  const int il = blockIdx.x / nj, i = pv.i0 + il, j = pv.i0 + blockIdx.x % nj;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const bool count = j >= i;
  const long long slot = (long long)blockIdx.x * gridDim.y + blockIdx.y;
  if (!GRAD && !count) {
    if (threadIdx.x < 2) part[2 * slot + threadIdx.x] = 0.0;
    return;
  }
  if (GRAD) {
    for (int c = threadIdx.x; c < v; c += 256) wv[c] = 0.0;
    __syncthreads();
  }
  double* P = pv.p + (long long)il * v * pv.ld + ((long long)j * v - pv.col0);
  const double eij = eps[i] + eps[j];
  const int nt = (v + PT - 1) / PT;
  double s0 = 0.0, s1 = 0.0;  // energy: os, ss; gradient: E, sum of W
  for (int tB = blockIdx.y; tB < nt; tB += gridDim.y) {
    const int b = tB * PT + tx;
    const double eb = b < v ? eps[o + b] : 0.0;
    double wcol = 0.0;
    for (int tA = 0; tA <= tB; ++tA) {
      double x[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int a = tA * PT + ty + 8 * r, bt = tB * PT + ty + 8 * r, at = tA * PT + tx;
        x[r] = a < v && b < v ? P[(long long)a * pv.ld + b] : 0.0;
        st[ty + 8 * r][tx] = bt < v && at < v ? P[(long long)bt * pv.ld + at] : 0.0;
      }
      __syncthreads();
      double y[4], g2[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) y[r] = st[tx][ty + 8 * r];
      const double half = tA == tB ? 0.5 : 1.0;
      double p0 = 0.0, p1 = 0.0;
      if (GRAD) __syncthreads();
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int a = tA * PT + ty + 8 * r;
        const bool live = a < v && b < v;
        double w = 0.0;
        g2[r] = 0.0;
        if (live) {
          const double rc = recip64((eps[o + a] + eb) - eij);
          if (GRAD) {
            const double tab = 2.0 * x[r] - y[r], tba = 2.0 * y[r] - x[r];
            const double s = fma(tab, x[r], tba * y[r]) * rc;
            const double rm = -2.0 * rc;
            p0 -= s;
            w = s * rc;
            P[(long long)a * pv.ld + b] = tab * rm;
            g2[r] = tba * rm;
            wcol = fma(half, w, wcol);
          } else {
            const double d = x[r] - y[r];
            p0 = fma(fma(x[r], x[r], y[r] * y[r]), rc, p0);
            p1 = fma(d * d, rc, p1);
          }
        }
        if (GRAD) st[ty + 8 * r][tx] = w;
      }
      s0 = fma(half, p0, s0);
      if (!GRAD) s1 = fma(half, p1, s1);
      __syncthreads();
      if (GRAD) {
        // row sums of W: eight lanes per row, warp ty owns rows 4 ty .. 4 ty + 3
        const int row = 4 * ty + (tx >> 3), c4 = (tx & 7) * 4;
        double rs = (st[row][c4] + st[row][c4 + 1]) + (st[row][c4 + 2] + st[row][c4 + 3]);
        rs += __shfl_xor_sync(0xffffffffu, rs, 1);
        rs += __shfl_xor_sync(0xffffffffu, rs, 2);
        rs += __shfl_xor_sync(0xffffffffu, rs, 4);
        const int a = tA * PT + row;
        if ((tx & 7) == 0 && a < v) wv[a] = fma(half, rs, wv[a]);
        __syncthreads();
        if (tA < tB) {  // G_ba back through shared memory
#pragma unroll
          for (int r = 0; r < 4; ++r) st[tx][ty + 8 * r] = g2[r];
          __syncthreads();
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int bt = tB * PT + ty + 8 * r, at = tA * PT + tx;
            if (bt < v && at < v) P[(long long)bt * pv.ld + at] = st[ty + 8 * r][tx];
          }
          __syncthreads();
        }
      }
    }
    if (GRAD) {  // column sums of W over the eight warps, fixed order
      st[ty][tx] = wcol;
      s1 += wcol;
      __syncthreads();
      if (ty == 0 && b < v) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += st[k][tx];
        wv[b] += t;
      }
      __syncthreads();
    }
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  if (tx == 0) {
    red[0][ty] = s0;
    red[1][ty] = s1;
  }
  __syncthreads();
  const double wij = i < j ? 2.0 : 1.0;  // ordered pairs
  if (GRAD) {
    if (count)
      for (int c = threadIdx.x; c < v; c += 256)
        if (wv[c] != 0.0) atomicAdd(&deps[o + c], wij * wv[c]);
    if (threadIdx.x == 0) {
      double es = 0.0, ws = 0.0;
      for (int k = 0; k < 8; ++k) {
        es += red[0][k];
        ws += red[1][k];
      }
      if (count) {
        atomicAdd(&deps[i], -wij * ws);
        atomicAdd(&deps[j], -wij * ws);
      }
      part[2 * slot] = count ? wij * es : 0.0;
      part[2 * slot + 1] = 0.0;
    }
  } else if (threadIdx.x < 2) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += red[threadIdx.x][k];
    part[2 * slot + threadIdx.x] = -wij * t;
  }
}

// The panel's diagonal (ia|ia) = sum_Q B^2 in FP64: 32 rows (i, a) per CTA, 32
// warps over Q, summed in a fixed order.  The digit products left out of a digit
// GEMM have no sign in general, but in a square d_4 d_4 has, and the integrals of
// real Gaussians are dominated by these elements (relative error of the energy,
// 768 auxiliary functions: 1e-15 without this kernel, 2e-16 with it).  Bound by
// HBM and the FP64 pipe alike: 8 bytes and one multiply-add per element of B.
__global__ void __launch_bounds__(1024) panel_diag_kernel(PanelView pv,
                                                          const double* __restrict__ bia, int X) {
  __shared__ double sm[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long r = blockIdx.x * 32ll + lane, R = (long long)pv.o * pv.v;
  const long long at = (long long)pv.i0 * pv.v + r;  // row (i, a) of B
  const bool live = r < (long long)pv.ni * pv.v;
  double s = 0.0;
  if (live) {
#pragma unroll 8
    for (int q = w; q < X; q += 32) {
      const double b = bia[(long long)q * R + at];
      s = fma(b, b, s);
    }
  }
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && live) {
    s = 0.0;
#pragma unroll
    for (int k = 0; k < 32; ++k) s += sm[k][lane];
    pv.p[r * pv.ld + (at - pv.col0)] = s;
  }
}

}  // namespace

PanelPlan panel_plan(int o, int v, int X, size_t budget) {
  PanelPlan p;
  const size_t per_i = (size_t)v * ((size_t)o * v + kDgColTile) * 8;
  p.ni = (int)std::max<size_t>(1, std::min<size_t>(o, budget / per_i));
  p.panel_bytes = per_i * p.ni;
  p.col_bytes = dgemm_tc_columns_bytes(o * v, X);
  if (p.col_bytes > kDgPlaneBytes + kDgPlaneBytes / 64) p.col_bytes = 0;  // (with the exponents)
  p.product_bytes = dgemm_tc_workspace(p.ni * v, p.col_bytes ? kDgColTile : o * v, X);
  long long n = 0;
  for (int i0 = 0; i0 < o; i0 += p.ni) n += (long long)std::min(p.ni, o - i0) * (o - i0);
  // CTAs per (i, j) block: one per column of tiles while that is a few million
  const int nt = (v + PT - 1) / PT;
  p.split = n * nt <= (1ll << 22) && nt <= 65535 ? nt : 1;
  p.partials = n * p.split;
  return p;
}

int panel_product(corr_context* c, int o, int v, int X, const double* bia, const DgColumns* cols,
                  int i0, int ni, double* panel, void* dws, PanelView* pv) {
  const int R = o * v;
  pv->p = panel;
  pv->col0 = (long long)i0 * v / kDgColTile * kDgColTile;
  pv->ld = R - pv->col0;
  pv->o = o;
  pv->v = v;
  pv->i0 = i0;
  pv->ni = ni;
  DgemmTc m;
  m.A = mat_view(bia + (size_t)i0 * v, 1, R);  // rows (i, a) of the block, over Q
  m.B = mat_view(bia + pv->col0, 1, R);
  m.C = out_view(panel, pv->ld, 1);
  m.M = ni * v;
  m.N = (int)pv->ld;
  m.K = X;
  m.alpha = 1.0;
  m.accumulate = false;
  m.a_lower = false;
  m.pre = cols;
  m.col0 = (int)pv->col0;
  CORR_TRY(dgemm_tc(c, m, dws));
  panel_diag_kernel<<<(unsigned)(((long long)ni * v + 31) / 32), 1024, 0, c->stream>>>(*pv, bia, X);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  return CORR_OK;
}

int launch_panel(corr_context* c, const PanelView& pv, const double* eps, double* deps,
                 double* part, int split, bool grad) {
  const dim3 grid((unsigned)(pv.ni * (pv.o - pv.i0)), (unsigned)split);
  // The W sums of a long virtual range go beyond the 48 KB that need no opt-in.  The
  // limit belongs to the kernel, not to a context: it is set to the largest nvir's,
  // the same for every caller.
  static bool attr[64] = {};
  if (grad && (c->device < 0 || c->device >= 64 || !attr[c->device])) {
    CORR_CUDA(cudaFuncSetAttribute(panel_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kPanelMaxNvir * 8));
    if (c->device >= 0 && c->device < 64) attr[c->device] = true;
  }
  if (grad)
    panel_kernel<true><<<grid, 256, (size_t)pv.v * 8, c->stream>>>(pv, eps, deps, part);
  else
    panel_kernel<false><<<grid, 256, 0, c->stream>>>(pv, eps, nullptr, part);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  return CORR_OK;
}

size_t energy_panel_bytes(int o, int v, int X) {
  const PanelPlan p = panel_plan(o, v, X, kPanelBudget);
  Carver w{nullptr, 0};
  w.take(p.panel_bytes);
  w.take(p.col_bytes);
  w.take(p.product_bytes);
  w.take((size_t)p.partials * 16);
  w.take(16);
  w.take((size_t)kReduceBlocks * 16);
  return w.used + 256;
}

int energy_from_panels(corr_context* c, Carver& w, int o, int v, int X, const double* bia,
                       const double* eps, double* out_e) {
  const PanelPlan p = panel_plan(o, v, X, kPanelBudget);
  double* panel = static_cast<double*>(w.take(p.panel_bytes));
  void* cws = w.take(p.col_bytes);
  void* dws = w.take(p.product_bytes);
  double* part = static_cast<double*>(w.take((size_t)p.partials * 16));
  unsigned* ticket = static_cast<unsigned*>(w.take(16));
  double* scratch = static_cast<double*>(w.take((size_t)kReduceBlocks * 16));
  DgColumns cols;
  if (p.col_bytes)
    CORR_TRY(dgemm_tc_slice_columns(c, mat_view(bia, 1, (long long)o * v), o * v, X, cws, &cols));
  long long np = 0;
  for (int i0 = 0; i0 < o; i0 += p.ni) {
    const int ni = std::min(p.ni, o - i0);
    PanelView pv;
    CORR_TRY(panel_product(c, o, v, X, bia, p.col_bytes ? &cols : nullptr, i0, ni, panel, dws,
                           &pv));
    CORR_TRY(launch_panel(c, pv, eps, nullptr, part + 2 * np, p.split, false));
    np += (long long)ni * (o - i0) * p.split;
  }
  CORR_CUDA(cudaMemsetAsync(ticket, 0, 16, c->stream));
  const int nr = launch_unit_reduce(part, (int)np, nullptr, out_e, scratch, ticket, c->stream);
  if (nr < 0) {
    set_error("energy reduction launch failed");
    return CORR_ERR_CUDA;
  }
  c->launches += nr;
  return CORR_OK;
}

}  // namespace corr
