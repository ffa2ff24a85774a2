// Blocked FP64 Cholesky factorisation of the RI metric and the triangular
// solve that applies it, for the energy-only RI pipeline.
//
// The RI-MP2 energy depends on the metric only through
//   (ia|jb) = sum_PQ (ia|P) [J^-1]_PQ (Q|jb),
// so any factor W with W^T W = J^-1 gives the same energy as the reference's
// symmetric J^-1/2 (src/POSTHF/ri.cc:50-69) whenever the reference cuts no
// eigenvalue.  With J = L L^T, W = L^-1 and B = L^-1 (P|ia) is one blocked
// forward substitution: m^2 ncols flops instead of the 2 m^2 ncols of the
// J^-1/2 product, and the factorisation costs m^3/3 instead of a full
// eigendecomposition.
//
// Whether the reference would cut an eigenvalue (lambda/lambda_max < tol) is
// decided by Sylvester's law of inertia: J - t I is positive definite exactly
// when every eigenvalue of J exceeds t.  With t = 10 tol ||J||_inf >= 10 tol
// lambda_max, a successful factorisation of J - t I certifies that no
// eigenvalue lies below tol lambda_max (the factor 10 covers the rounding of
// either factorisation, ~m eps ||J||).  Without the certificate the caller
// falls back to the eigendecomposition (jacobi.cu).
//
// Layout: row-major m x m.  Block size 64: one CTA factors the diagonal block
// in shared memory and also inverts it; the panel below is L21 = A21 L11^-T
// and the trailing update A22 -= L21 L21^T (gemm_fp64.cu, or dgemm_tc.cu where
// the context allows it and the product is large).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "dgemm_tc.h"
#include "fp64_approx.cuh"
#include "gemm_fp64.h"
#include "kernels.h"

namespace corr {

namespace {

constexpr int NB = 64;

// A = J - shift I (m x m), Lm = 0.
__global__ void chol_init(const double* __restrict__ J, int m, double shift,
                          double* __restrict__ A, double* __restrict__ Lm) {
  const long long mm = (long long)m * m;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < mm;
       e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e / m), y = (int)(e % m);
    A[e] = J[e] - (x == y ? shift : 0.0);
    Lm[e] = 0.0;
  }
}

// One CTA: factor the nb x nb diagonal block at (k, k) of A (lower triangle
// read), write L_kk into Lm and its inverse into Linv (leading dimension ldi;
// `pad`: zeros up to NB x NB).  A pivot that is not positive (or not finite)
// sets *fail.
//
// The block is eliminated in place with the identity: with A = U D U^T (U unit
// lower triangular), step c subtracts q_i v_j from row i > c, q_i = M_ic / d_c,
// v_j = M_jc for j > c and the finished row c of U^-1 for j <= c, so the lower
// triangle ends as U^-1 while the columns q of U go to shared memory.  Row i
// has i + 1 live elements at every step: warp w keeps rows w, w + 8, ... in
// registers, lane = column, and each step is one barrier.  L = U D^1/2 and
// L^-1 = D^-1/2 U^-1 at the end.
//
// Bound by one SM's FP64 pipe (16 clocks per warp instruction: 57k clocks for
// the updates of a 64 x 64 block, 28 us) and the chain of pivots (reciprocal,
// multiplier, update: about 600 clocks a step).  60 us; 150 us with a square root,
// divisions and three barriers per column and the inverse in a second pass.
__global__ void __launch_bounds__(256) chol_diag(const double* __restrict__ A, int m, int k,
                                                 int nb, double* __restrict__ Lm,
                                                 double* __restrict__ Linv, int ldi, int pad,
                                                 int* fail) {
  __shared__ double Us[NB][NB + 1];
  __shared__ double col[2][NB], row[2][NB], rd[2], dv[NB], sq[NB], rs[NB];
  __shared__ int bad;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) bad = 0;
  // M[i][lane] and M[i][lane + 32] of rows i = warp + 8 r; rows beyond nb are
  // the identity
  double m0[8], m1[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = warp + 8 * r, j0 = lane, j1 = lane + 32;
    m0[r] = i < nb && j0 <= i ? A[(size_t)(k + i) * m + k + j0] : (i == j0 ? 1.0 : 0.0);
    m1[r] = i < nb && j1 <= i ? A[(size_t)(k + i) * m + k + j1] : (i == j1 ? 1.0 : 0.0);
  }
  // pivot of row c (register index r) and its reciprocal, by the row's warp
  double pd = 1.0, pr = 1.0;
  auto pivot = [&](double mc, int cl) {
    pd = __shfl_sync(0xffffffffu, mc, cl);
    const int ex = (__double2hiint(pd) >> 20);  // sign and exponent
    if (ex <= 0 || ex >= 0x7FF) {               // not positive, normal and finite
      pd = 1.0;
      bad = 1;
    }
    pr = recip64(pd);
  };
  __syncthreads();
  if (warp == 0) pivot(m0[0], 0);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
#pragma unroll 1
    for (int w = 0; w < 8; ++w) {
      const int c = 8 * kk + w, b = w & 1, cl = c & 31;
      if (lane == cl) {  // column c of the rows from c on
#pragma unroll
        for (int r = kk; r < 8; ++r) col[b][warp + 8 * r] = kk < 4 ? m0[r] : m1[r];
      }
      if (warp == w) {  // row c, its pivot and the pivot's reciprocal
        row[b][lane] = m0[kk];
        row[b][lane + 32] = m1[kk];
        if (lane == 0) {
          rd[b] = pr;
          dv[c] = pd;
        }
      }
      __syncthreads();
      const int j1 = lane + 32;
      const double v0 = lane < c ? row[b][lane] : (lane == c ? 1.0 : col[b][lane]);
      const double v1 = j1 < c ? row[b][j1] : (j1 == c ? 1.0 : col[b][j1]);
      // lane r: q of row warp + 8 r
      const int iq = warp + 8 * (lane & 7);
      const double q = iq > c ? col[b][iq] * rd[b] : 0.0;
      if (lane < 8 && iq > c) Us[iq][c] = q;
      auto update = [&](int r) {  // r a constant after unrolling
        const double qr = __shfl_sync(0xffffffffu, q, r);
        if (kk < 4) {
          m0[r] = fma(-qr, v0, lane == cl ? 0.0 : m0[r]);
          if (r >= 4) m1[r] = fma(-qr, v1, m1[r]);
        } else {
          m0[r] = fma(-qr, v0, m0[r]);
          m1[r] = fma(-qr, v1, lane == cl ? 0.0 : m1[r]);
        }
      };
      // the next pivot's row first, so that its reciprocal is under way while
      // the pipe works on the other rows
      if (w < 7) {
        if (warp > w) update(kk);  // rows up to c are finished
        if (warp == w + 1) pivot(kk < 4 ? m0[kk] : m1[kk], (c + 1) & 31);
#pragma unroll
        for (int r = kk + 1; r < 8; ++r) update(r);
      } else if (kk < 7) {
        constexpr int last = 7;
        const int rn = kk < last ? kk + 1 : last;
        update(rn);
        if (warp == 0) pivot(kk + 1 < 4 ? m0[rn] : m1[rn], (c + 1) & 31);
#pragma unroll
        for (int r = kk + 2; r < 8; ++r) update(r);
      }
    }
  }
  __syncthreads();
  if (t < NB) {
    sq[t] = sqrt(dv[t]);
    rs[t] = 1.0 / sq[t];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = warp + 8 * r;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + 32 * h;
      const bool live = i < nb && j < nb;
      const double x = live && j <= i ? (j == i ? rs[i] : (h ? m1[r] : m0[r]) * rs[i]) : 0.0;
      if (live || pad) Linv[(size_t)i * ldi + j] = x;
      if (live)
        Lm[(size_t)(k + i) * m + k + j] = j < i ? Us[i][j] * sq[j] : (j == i ? sq[i] : 0.0);
    }
  }
  if (t == 0 && bad) atomicExch(fail, 1);
}

// max_r sum_c |J[r][c]| (one warp per row; non-negative doubles order as
// their bit patterns).
__global__ void norm_inf_kernel(const double* __restrict__ J, int m,
                                unsigned long long* __restrict__ out) {
  const int warps = (int)(gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < m; r += warps) {
    double s = 0.0;
    for (int c = lane; c < m; c += 32) s += fabs(J[(size_t)r * m + c]);
    s = warp_sum(s);
    if (lane == 0) atomicMax(out, (unsigned long long)__double_as_longlong(s));
  }
}

// max_c sum_r |X[r][c]|: a block of 32 warps per 32 columns, fixed order.
__global__ void __launch_bounds__(1024) norm_one_kernel(const double* __restrict__ X, int m,
                                                        unsigned long long* __restrict__ out) {
  __shared__ double sm[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int cidx = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (cidx < m)
#pragma unroll 4
    for (int r = w; r < m; r += 32) s += fabs(X[(size_t)r * m + cidx]);
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && cidx < m) {
    s = 0.0;
    for (int q = 0; q < 32; ++q) s += sm[q][lane];
    atomicMax(out, (unsigned long long)__double_as_longlong(s));
  }
}

}  // namespace

size_t chol_workspace_bytes(int m) {
  const int nblk = (m + NB - 1) / NB;
  return (size_t)2 * m * m * 8 + (size_t)nblk * NB * NB * 8 + 3 * 256;
}

int chol_norm_inf(corr_context* c, void* scratch, const double* J, int m, double* out) {
  unsigned long long* d = static_cast<unsigned long long*>(scratch);
  CORR_CUDA(cudaMemsetAsync(d, 0, sizeof(*d), c->stream));
  norm_inf_kernel<<<(m + 7) / 8, 256, 0, c->stream>>>(J, m, d);
  CORR_CUDA(cudaGetLastError());
  unsigned long long h = 0;
  CORR_CUDA(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  CORR_CUDA(cudaStreamSynchronize(c->stream));
  c->launches += 1;
  double v;
  memcpy(&v, &h, sizeof(v));
  *out = v;
  return CORR_OK;
}

// tc_ws: when non-null, the panel and trailing products run on the
// FP64-accurate digit GEMM (dgemm_tc.cu) with that workspace
// (dgemm_tc_workspace(m, m, NB) bytes); else on the FP64 GEMM.
int chol_factor_device(corr_context* c, void* ws, const double* J, int m, double shift,
                       double** Lm_out, double** Linv_out, bool* ok, void* tc_ws) {
  const int nblk = (m + NB - 1) / NB;
  Carver w{ws, 0};
  double* A = static_cast<double*>(w.take((size_t)m * m * 8));
  double* Lm = static_cast<double*>(w.take((size_t)m * m * 8));
  double* Linv = static_cast<double*>(w.take((size_t)nblk * NB * NB * 8));
  int* fail = static_cast<int*>(w.take(sizeof(int)));
  cudaStream_t s = c->stream;
  CORR_CUDA(cudaMemsetAsync(fail, 0, sizeof(int), s));
  const int ig = (int)std::min<long long>(((long long)m * m + 255) / 256, 4096);
  chol_init<<<ig, 256, 0, s>>>(J, m, shift, A, Lm);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  for (int b = 0; b < nblk; ++b) {
    const int k = b * NB, nb = std::min(NB, m - k), rem = m - k - nb;
    double* Li = Linv + (size_t)b * NB * NB;
    chol_diag<<<1, 256, 0, s>>>(A, m, k, nb, Lm, Li, NB, 1, fail);
    CORR_CUDA(cudaGetLastError());
    c->launches += 1;
    if (rem == 0) break;
    const double* P = Lm + (size_t)(k + nb) * m + k;
    {
      // L21 = A21 L11^-T (few enough multiply-adds for the FP64 pipe)
      GemmF64 g = gemm_args(A + (size_t)(k + nb) * m + k, Li, Lm + (size_t)(k + nb) * m + k, rem,
                            nb, nb, m, NB, m, 0, 1);
      CORR_TRY(gemm_f64(g, &c->dres->status, s));
      c->launches += 1;
    }
    if (tc_ws && (double)rem * rem * nb >= 1e7) {
      DgemmTc g;
      g.A = mat_view(P, m, 1);
      g.B = mat_view(P, m, 1);
      g.C = out_view(A + (size_t)(k + nb) * m + k + nb, m, 1);
      g.M = rem;
      g.N = rem;
      g.K = nb;
      g.alpha = -1.0;
      g.accumulate = true;
      g.a_lower = false;
      CORR_TRY(dgemm_tc(c, g, tc_ws));  // A22 -= L21 L21^T
    } else {
      // A22 -= L21 L21^T
      GemmF64 u = gemm_args(P, P, A + (size_t)(k + nb) * m + k + nb, rem, rem, nb, m, m, m, 0, 1);
      u.alpha = -1.0;
      u.beta = 1.0;
      CORR_TRY(gemm_f64(u, &c->dres->status, s));
      c->launches += 1;
    }
  }
  int h = 0;
  CORR_CUDA(cudaMemcpyAsync(&h, fail, sizeof(int), cudaMemcpyDeviceToHost, s));
  CORR_CUDA(cudaStreamSynchronize(s));
  *ok = (h == 0);
  *Lm_out = Lm;
  *Linv_out = Linv;
  return CORR_OK;
}

int chol_solve_device(corr_context* c, const double* Lm, const double* Linv, int m, double* P,
                      long long ncols, double* out) {
  const int nblk = (m + NB - 1) / NB;
  cudaStream_t s = c->stream;
  for (int b = 0; b < nblk; ++b) {
    const int r0 = b * NB, nb = std::min(NB, m - r0);
    double* Pi = P + (size_t)r0 * ncols;
    if (r0 > 0) {
      // P_i -= L[r0:r0+nb, 0:r0] B[0:r0, :]
      GemmF64 g = gemm_args(Lm + (size_t)r0 * m, out, Pi, nb, (int)ncols, r0, m, ncols, ncols, 0,
                            0);
      g.alpha = -1.0;
      g.beta = 1.0;
      CORR_TRY(gemm_f64(g, &c->dres->status, s));
    }
    // B_i = L_ii^-1 P_i
    CORR_TRY(gemm_f64(gemm_args(Linv + (size_t)b * NB * NB, Pi, out + (size_t)r0 * ncols, nb,
                                (int)ncols, nb, NB, ncols, ncols, 0, 0),
                      &c->dres->status, s));
    c->launches += (r0 > 0) ? 2 : 1;
  }
  return CORR_OK;
}

// L (into *Lm_out) and X = L^-1 of J - shift I together, by recursive splitting
// on 64-aligned halves: factor and invert the first half, L21 = A21 X11^T,
// A22 -= L21 L21^T, the second half, X21 = -X22 (L21 X11).  Against the
// right-looking factorisation followed by an inversion this has a fraction of
// the dependent launches, and its products have K up to m / 2 instead of 64.
// ws: chol_workspace_bytes(m); T: scratch of m * m doubles; tc_ws: digit-GEMM
// workspace for (m, m, m).  Products below 1e7 multiply-adds run on the FP64
// pipe.  m = 1520: 3.7 ms of kernels (6.9 ms).
int chol_factor_inverse_device(corr_context* c, void* ws, const double* J, int m, double shift,
                               double* X, double* T, double** Lm_out, bool* ok, void* tc_ws) {
  Carver w{ws, 0};
  double* A = static_cast<double*>(w.take((size_t)m * m * 8));
  double* Lm = static_cast<double*>(w.take((size_t)m * m * 8));
  int* fail = static_cast<int*>(w.take(sizeof(int)));
  cudaStream_t s = c->stream;
  CORR_CUDA(cudaMemsetAsync(fail, 0, sizeof(int), s));
  CORR_CUDA(cudaMemsetAsync(X, 0, (size_t)m * m * 8, s));
  const int ig = (int)std::min<long long>(((long long)m * m + 255) / 256, 4096);
  chol_init<<<ig, 256, 0, s>>>(J, m, shift, A, Lm);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  // C (M x N) = alpha A op(B) (+ C), all with leading dimension m but ldb, ldc
  auto product = [&](const double* pa, const double* pb, int tb, long long ldb, double* pc,
                     long long ldc, int M, int N, int K, double alpha, bool add,
                     bool a_lower) -> int {
    if ((double)M * N * K < 1e7) {
      GemmF64 g = gemm_args(pa, pb, pc, M, N, K, m, ldb, ldc, 0, tb);
      g.alpha = alpha;
      g.beta = add ? 1.0 : 0.0;
      c->launches += 1;
      return gemm_f64(g, &c->dres->status, s);
    }
    DgemmTc g;
    g.A = mat_view(pa, m, 1);
    g.B = tb ? mat_view(pb, ldb, 1) : mat_view(pb, 1, ldb);
    g.C = out_view(pc, ldc, 1);
    g.M = M;
    g.N = N;
    g.K = K;
    g.alpha = alpha;
    g.accumulate = add;
    g.a_lower = a_lower;
    return dgemm_tc(c, g, tc_ws);
  };
  // steps of the recursion in order: a leaf, or the products before / after the
  // second half
  struct Step {
    int r0, n, stage;
  };
  std::vector<Step> stack{{0, m, 0}};
  while (!stack.empty()) {
    const Step st = stack.back();
    stack.pop_back();
    const int n1 = NB * (((st.n + NB - 1) / NB + 1) / 2), n2 = st.n - n1;
    const int r0 = st.r0, r1 = r0 + n1;
    auto at = [&](double* p, int r, int q) { return p + (size_t)r * m + q; };
    if (st.stage == 0) {
      if (st.n <= NB) {
        chol_diag<<<1, 256, 0, s>>>(A, m, r0, st.n, Lm, at(X, r0, r0), m, 0, fail);
        CORR_CUDA(cudaGetLastError());
        c->launches += 1;
        continue;
      }
      stack.push_back({r0, st.n, 2});
      stack.push_back({r1, n2, 0});
      stack.push_back({r0, st.n, 1});
      stack.push_back({r0, n1, 0});
    } else if (st.stage == 1) {
      CORR_TRY(product(at(A, r1, r0), at(X, r0, r0), 1, m, at(Lm, r1, r0), m, n2, n1, n1, 1.0,
                       false, false));
      CORR_TRY(product(at(Lm, r1, r0), at(Lm, r1, r0), 1, m, at(A, r1, r1), m, n2, n2, n1, -1.0,
                       true, false));
    } else {
      CORR_TRY(product(at(Lm, r1, r0), at(X, r0, r0), 0, m, T, n1, n2, n1, n1, 1.0, false, false));
      CORR_TRY(product(at(X, r1, r1), T, 0, n1, at(X, r1, r0), m, n2, n1, n2, -1.0, false, true));
    }
  }
  int h = 0;
  CORR_CUDA(cudaMemcpyAsync(&h, fail, sizeof(int), cudaMemcpyDeviceToHost, s));
  CORR_CUDA(cudaStreamSynchronize(s));
  *ok = (h == 0);
  *Lm_out = Lm;
  return CORR_OK;
}

// ||X||_1 ||X||_inf of an m x m matrix (scratch: 16 bytes of device memory).
int chol_norm_one_inf(corr_context* c, void* scratch, const double* X, int m, double* out) {
  unsigned long long* d = static_cast<unsigned long long*>(scratch);
  CORR_CUDA(cudaMemsetAsync(d, 0, 2 * sizeof(*d), c->stream));
  norm_one_kernel<<<(m + 31) / 32, 1024, 0, c->stream>>>(X, m, d);
  norm_inf_kernel<<<(m + 7) / 8, 256, 0, c->stream>>>(X, m, d + 1);
  CORR_CUDA(cudaGetLastError());
  unsigned long long h[2] = {0, 0};
  CORR_CUDA(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  CORR_CUDA(cudaStreamSynchronize(c->stream));
  c->launches += 2;
  double v[2];
  memcpy(v, h, sizeof(v));
  *out = v[0] * v[1];
  return CORR_OK;
}

}  // namespace corr
