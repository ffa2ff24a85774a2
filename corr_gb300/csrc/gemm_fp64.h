// FP64 GEMM building block (gemm_fp64.cu) and the FP64 hot-path helpers built
// on it (transforms.cu).
#pragma once

#include <cuda_runtime.h>

#include "abi_internal.h"

namespace corr {

struct GemmF64 {
  const double* A;
  const double* B;
  double* C;
  int M, N, K;
  long long lda, ldb, ldc;
  long long sa, sb, sc;  // batch strides (elements), 0 = shared operand
  int batch;
  int ta, tb;
  double alpha, beta;
};

// Enqueue C = alpha op(A) op(B) + beta C on stream s.
int gemm_f64(const GemmF64& g, int* status, cudaStream_t s);

// The plain form's product C = alpha op(A) op(B) (one matrix, beta = 0): on the
// digit GEMM of dgemm_tc.cu where that is faster and the context does not ask
// for the FP64 pipe (corr_set_fp64_strict), else gemm_f64.  ws:
// gemm_plain_workspace bytes.  Values out of the digit GEMM's range raise
// kStatusNeedFp64.
size_t gemm_plain_workspace(const corr_context* c, long long M, long long N, long long K);
int gemm_plain(corr_context* c, const GemmF64& g, void* ws);
// The rule: from 1e7 multiply-adds on, where the FP64 pipe takes 17 us at its
// full rate of 5.9e5 per us, the slicing (three launches, about 10 us) and one
// round of digit-GEMM tiles are the shorter way: 200^3 takes 18 us against 33 us,
// 256^3 42 us against 34 us, 128^3 8 us against 28 us.
inline bool digits_pay(const corr_context* c, long long M, long long N, long long K) {
  return !c->fp64_strict && (double)M * N * K >= 1e7 && M <= 0x7fffff00LL && N <= 0x7fffff00LL;
}

inline GemmF64 gemm_args(const double* A, const double* B, double* C, int M, int N, int K,
                         long long lda, long long ldb, long long ldc, int ta, int tb) {
  GemmF64 g;
  g.A = A;
  g.B = B;
  g.C = C;
  g.M = M;
  g.N = N;
  g.K = K;
  g.lda = lda;
  g.ldb = ldb;
  g.ldc = ldc;
  g.sa = g.sb = g.sc = 0;
  g.batch = 1;
  g.ta = ta;
  g.tb = tb;
  g.alpha = 1.0;
  g.beta = 0.0;
  return g;
}

}  // namespace corr
