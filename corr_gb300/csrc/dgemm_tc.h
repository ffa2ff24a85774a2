// FP64-accurate GEMM on the tensor cores (dgemm_tc.cu): exact digit slicing
// of both FP64 operands, integer-exact level sums on tcgen05 (kind::f16, BF16
// digits, FP32 accumulation in TMEM), integer recombination to FP64.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "abi_internal.h"

namespace corr {

// An FP64 matrix read as `rows` x K: element (r, k) at
//   p[(r / rdiv) * rs_hi + (r % rdiv) * rs_lo + k * ks]
// (rdiv = rows, rs_hi = 0 for a plain strided matrix; a two-level row index
// for row sets such as (P, nu) of a 3-index tensor).
struct MatView {
  const double* p;
  long long rs_hi, rs_lo, ks, rdiv;
};
// Output element (m, n) at p[(m / rdiv) * rs_hi + (m % rdiv) * rs_lo + n * cs].
struct OutView {
  double* p;
  long long rs_hi, rs_lo, cs, rdiv;
};

inline MatView mat_view(const double* p, long long rs, long long ks) {
  return MatView{p, 0, rs, ks, 1LL << 62};
}
inline OutView out_view(double* p, long long rs, long long cs) {
  return OutView{p, 0, rs, cs, 1LL << 62};
}

// A column operand sliced once for several products (dgemm_tc_slice_columns).
struct DgColumns {
  const uint16_t* planes = nullptr;
  const int* e = nullptr;
  int rows_pad = 0;
};

// C[m][n] = alpha sum_k A(m, k) B(n, k) (+ C[m][n] when accumulate), m < M,
// n < N, k < K.  a_lower: A(m, k) == 0 for k > m (skipped).  Inputs finite;
// in a plain-form call (corr_context::digit_guard) an operand with a value
// outside the splitting's range (not finite, or a row whose largest magnitude
// in 512 of K is below 2^-958) raises kStatusNeedFp64 in the context's status word.
struct DgemmTc {
  MatView A, B;
  OutView C;
  int M, N, K;
  double alpha;
  bool accumulate;
  bool a_lower;
  // B already sliced: column n of this product is row col0 + n of `pre` (col0
  // a multiple of kDgColTile), and B is not read.
  const DgColumns* pre = nullptr;
  int col0 = 0;
};
constexpr int kDgColTile = 64;
// Digit planes of an operand at a time (16 bytes per element); a product whose
// operand takes more runs in blocks of its rows or columns.
constexpr size_t kDgPlaneBytes = (size_t)1 << 30;

// Device workspace of one dgemm_tc call (bytes).
size_t dgemm_tc_workspace(int M, int N, int K);
// Enqueue on the context stream; ws holds dgemm_tc_workspace(M, N, K) bytes.
int dgemm_tc(corr_context* c, const DgemmTc& g, void* ws);

// The digit planes of a column operand of `rows` rows over K, kept in `ws`
// (dgemm_tc_columns_bytes) while *out is used.
size_t dgemm_tc_columns_bytes(int rows, int K);
int dgemm_tc_slice_columns(corr_context* c, const MatView& v, int rows, int K, void* ws,
                           DgColumns* out);

}  // namespace corr
