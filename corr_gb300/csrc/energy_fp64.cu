// Plain FP64 fused RI-MP2 energy on the FP64 tensor path (mma.sync m8n8k4 f64).
//
// Work unit = (occupied pair i<=j, virtual tile pair A<=B).  A unit forms two
// 64x64 tiles of the exchange-paired integrals
//   D1[a][b] = (ia|jb) = sum_Q B^Q_ia B^Q_jb          (a in A, b in B)
//   D2[a][b] = (ib|ja) = sum_Q B^Q_ja B^Q_ib
// in registers and folds them straight into the energy:
//   E_OS -= f w (D1^2 + D2^2) / D,   E_SS -= f w (D1 - D2)^2 / D,
// D = e_a + e_b - e_i - e_j, f = 2 if A<B else 1, w = 1 if i<j else 1/2.
// Summed over units this is exactly the reference's double sum over ordered
// (i,j) and all (a,b) (can_mp2.cc:82-97): the (j,i) term equals the (i,j) term
// with a and b swapped, and the (b,a) element of a pair pairs with (a,b).
// No (ia|jb) value ever reaches global memory.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace corr {

namespace {

constexpr int T = kF64Tile;  // 64
constexpr int KB = 16;       // Q rows per step
constexpr int LD = T + 4;    // padded smem row (doubles): conflict-free fragment loads

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(128) energy_fp64_kernel(const double* __restrict__ bia,
                                                          const double* __restrict__ eps,
                                                          EnergyShape sh,
                                                          double* __restrict__ partials) {
  __shared__ double s_iA[KB][LD], s_jB[KB][LD], s_jA[KB][LD], s_iB[KB][LD];
  __shared__ double red[2][4];
  const int o = sh.nocc, v = sh.nvir, X = sh.naux;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int g = lane >> 2, t = lane & 3;
  const long long rowQ = (long long)o * v;  // stride between Q rows

  double tot_os = 0.0, tot_ss = 0.0;

  for (long long u = blockIdx.x; u < sh.nunits; u += gridDim.x) {
    int p = (int)(u / sh.ntpairs), tp = (int)(u % sh.ntpairs);
    int i, j, A, B;
    pair_decode(p, o, &i, &j);
    tpair_decode(tp, sh.ntiles, &A, &B);
    const int A0 = A * T, B0 = B * T;

    double acc1[4][4][2], acc2[4][4][2];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        acc1[mi][ni][0] = acc1[mi][ni][1] = 0.0;
        acc2[mi][ni][0] = acc2[mi][ni][1] = 0.0;
      }

    for (int q0 = 0; q0 < X; q0 += KB) {
#pragma unroll
      for (int e = 0; e < (KB * T) / 128; ++e) {
        int idx = tid + 128 * e;
        int r = idx / T, c = idx % T;
        int q = q0 + r;
        bool qok = q < X;
        const double* base = bia + (long long)q * rowQ;
        int a = A0 + c, b = B0 + c;
        s_iA[r][c] = (qok && a < v) ? base[(long long)i * v + a] : 0.0;
        s_jA[r][c] = (qok && a < v) ? base[(long long)j * v + a] : 0.0;
        s_jB[r][c] = (qok && b < v) ? base[(long long)j * v + b] : 0.0;
        s_iB[r][c] = (qok && b < v) ? base[(long long)i * v + b] : 0.0;
      }
      __syncthreads();
#pragma unroll
      for (int k0 = 0; k0 < KB; k0 += 4) {
        double a1[4], a2[4], b1[4], b2[4];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
          a1[mi] = s_iA[k0 + t][wm * 32 + mi * 8 + g];
          a2[mi] = s_jA[k0 + t][wm * 32 + mi * 8 + g];
        }
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          b1[ni] = s_jB[k0 + t][wn * 32 + ni * 8 + g];
          b2[ni] = s_iB[k0 + t][wn * 32 + ni * 8 + g];
        }
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) {
            dmma(acc1[mi][ni], a1[mi], b1[ni]);
            dmma(acc2[mi][ni], a2[mi], b2[ni]);
          }
      }
      __syncthreads();
    }

    // fused epilogue: denominators and pair energies in FP64
    const double ei = eps[i], ej = eps[j];
    double los = 0.0, lss = 0.0;
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      int a = A0 + wm * 32 + mi * 8 + g;
      if (a >= v) continue;
      double ea = eps[o + a];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          int b = B0 + wn * 32 + ni * 8 + 2 * t + e;
          if (b >= v) continue;
          double den = ((ea + eps[o + b]) - ei) - ej;
          double d1 = acc1[mi][ni][e], d2 = acc2[mi][ni][e];
          double r = 1.0 / den;
          los += (d1 * d1 + d2 * d2) * r;
          double df = d1 - d2;
          lss += df * df * r;
        }
    }
    double fw = (A < B ? 2.0 : 1.0) * (i < j ? 1.0 : 0.5);
    tot_os -= fw * los;
    tot_ss -= fw * lss;
  }

  tot_os = warp_sum(tot_os);
  tot_ss = warp_sum(tot_ss);
  if (lane == 0) {
    red[0][warp] = tot_os;
    red[1][warp] = tot_ss;
  }
  __syncthreads();
  if (tid == 0) {
    partials[2 * blockIdx.x] = (red[0][0] + red[0][1]) + (red[0][2] + red[0][3]);
    partials[2 * blockIdx.x + 1] = (red[1][0] + red[1][1]) + (red[1][2] + red[1][3]);
  }
}

// The same sums on 8 x 8 tiles; S warps (4 or 1) share a unit and split its Q;
// fragments straight from global memory (every unit of the same occupied pair
// reads the same rows: L1/L2).  For small problems: a 64 x 64 tile costs the
// FP64 pipe (two FMAs per clock per SM) 2 * 4096 FMAs per Q however few
// virtuals there are, and there are few units to spread over the SMs.
// nocc=5 nvir=19 naux=76, 90 units of 8 x 8 instead of 15 of 64 x 64: 7.0 us
// instead of 210 us (14.8 us with S = 1, a chain of 19 steps).  With more units
// than CTAs the FP64 pipe is the bound and S = 1 saves the exchange (nocc=9
// nvir=64 naux=31: 21.3 us against 27.9 us).
constexpr int ST = 8;

template <int S>
__global__ void __launch_bounds__(128) energy_fp64_small_kernel(const double* __restrict__ bia,
                                                                const double* __restrict__ eps,
                                                                EnergyShape sh,
                                                                double* __restrict__ partials) {
  __shared__ double part[4][4][32];
  __shared__ double red[4][2];
  const int o = sh.nocc, v = sh.nvir, X = sh.naux;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int sub = warp % S;  // this warp's part of its unit's Q
  const long long rowQ = (long long)o * v;
  double tot_os = 0.0, tot_ss = 0.0;
  for (long long u0 = blockIdx.x * (4ll / S); u0 < sh.nunits; u0 += gridDim.x * (4ll / S)) {
    const long long u = u0 + warp / S;
    if (S == 1 && u >= sh.nunits) break;
    int i, j, A, B;
    pair_decode((int)(u / sh.ntpairs), o, &i, &j);
    tpair_decode((int)(u % sh.ntpairs), sh.ntiles, &A, &B);
    const int ra = A * ST + g, rb = B * ST + g;
    const bool la = ra < v, lb = rb < v;
    double acc1[2] = {0.0, 0.0}, acc2[2] = {0.0, 0.0};
#pragma unroll 4
    for (int q0 = 4 * sub; q0 < X; q0 += 4 * S) {
      const int q = q0 + t;
      const bool lq = q < X;
      const double* bi = bia + (long long)q * rowQ + (long long)i * v;
      const double* bj = bia + (long long)q * rowQ + (long long)j * v;
      const double a1 = lq && la ? bi[ra] : 0.0, b1 = lq && lb ? bj[rb] : 0.0;
      const double a2 = lq && la ? bj[ra] : 0.0, b2 = lq && lb ? bi[rb] : 0.0;
      dmma(acc1, a1, b1);
      dmma(acc2, a2, b2);
    }
    double d[4] = {acc1[0], acc1[1], acc2[0], acc2[1]};
    if (S > 1) {
#pragma unroll
      for (int k = 0; k < 4; ++k) part[warp][k][lane] = d[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 4; ++k)
        d[k] = (part[0][k][lane] + part[1][k][lane]) + (part[2][k][lane] + part[3][k][lane]);
    }
    if (sub == 0 && la) {
      double los = 0.0, lss = 0.0;
      const double eai = eps[o + ra];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int b = B * ST + 2 * t + e;
        if (b >= v) continue;
        const double r = 1.0 / (((eai + eps[o + b]) - eps[i]) - eps[j]);
        const double df = d[e] - d[2 + e];
        los += (d[e] * d[e] + d[2 + e] * d[2 + e]) * r;
        lss += df * df * r;
      }
      const double fw = (A < B ? 2.0 : 1.0) * (i < j ? 1.0 : 0.5);
      tot_os -= fw * los;
      tot_ss -= fw * lss;
    }
    if (S > 1) __syncthreads();
  }
  tot_os = warp_sum(tot_os);
  tot_ss = warp_sum(tot_ss);
  if (lane == 0) {
    red[warp][0] = tot_os;
    red[warp][1] = tot_ss;
  }
  __syncthreads();
  if (threadIdx.x < 2)
    partials[2 * blockIdx.x + threadIdx.x] = (red[0][threadIdx.x] + red[1][threadIdx.x]) +
                                             (red[2][threadIdx.x] + red[3][threadIdx.x]);
}

}  // namespace

int launch_energy_fp64(const double* bia, const double* eps, const EnergyShape& sh,
                       double* partials, int grid, int sms, cudaStream_t s) {
  // Small tiles when they give the busiest SM at most half the FMAs and the
  // 64 x 64 units would not fill four rounds of it.
  const EnergyShape s8 = make_energy_shape(sh.nocc, sh.nvir, sh.naux, ST);
  const long long w64 = (sh.nunits + sms - 1) / sms * T * T;
  const long long w8 = (s8.nunits + sms - 1) / sms * ST * ST;
  if (sh.nunits <= 4ll * sms && 2 * w8 <= w64) {
    const bool split = s8.nunits <= 2ll * sms;
    const int sgrid = (int)std::min<long long>(split ? s8.nunits : (s8.nunits + 3) / 4, 2ll * sms);
    if (split)
      energy_fp64_small_kernel<4><<<sgrid, 128, 0, s>>>(bia, eps, s8, partials);
    else
      energy_fp64_small_kernel<1><<<sgrid, 128, 0, s>>>(bia, eps, s8, partials);
    return cudaGetLastError() == cudaSuccess ? sgrid : -1;
  }
  energy_fp64_kernel<<<grid, 128, 0, s>>>(bia, eps, sh, partials);
  return cudaGetLastError() == cudaSuccess ? grid : -1;
}

}  // namespace corr
