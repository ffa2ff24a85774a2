// Diagnostics.
//
// corr_selftest_wait_timeout: the bounded-wait path of the kernels, exercised on
// purpose.
// Every mbarrier wait of the tcgen05 kernels gives up after a time limit,
// raises CORR_ERR_DEVICE_TIMEOUT in the call's status word and lets the CTA
// wind down, so a lost arrival never hangs the GPU.  This entry point runs
// that path: one CTA waits, with the same primitive, on an mbarrier phase that
// nothing completes, for a caller-chosen limit.  No fault, trap or unbounded
// loop is involved; the context stays usable afterwards.
//
// corr_selftest_fp64: the FP64 functions of fp64_approx.cuh, one argument per
// thread.
//
// corr_selftest_factor: the Cholesky factor with its inverse (chol.cu) as the
// precision forms of the 3-index pipeline take it, which otherwise shows only in
// energies that their own digits limit to 1e-8.
#include "abi_internal.h"
#include "common.cuh"
#include "dgemm_tc.h"
#include "fp64_approx.cuh"

namespace corr {
size_t chol_workspace_bytes(int m);
int chol_factor_inverse_device(corr_context* c, void* ws, const double* J, int m, double shift,
                               double* X, double* T, double** Lm_out, bool* ok, void* tc_ws);
namespace {

__global__ void wait_selftest_kernel(unsigned long long limit_ns, int* status) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);  // one arrival expected; none is ever made
    abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait_for(&bar, 0, &abort_flag, status, limit_ns);
}

__global__ void fp64_selftest_kernel(int which, long long n, const double* __restrict__ x,
                                     double* __restrict__ out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    out[k] = which ? rsqrt64(x[k]) : recip64(x[k]);
}

}  // namespace
}  // namespace corr

using namespace corr;

extern "C" {

int corr_selftest_wait_timeout(corr_context* c, int limit_ms) {
  CORR_CHECK_ARG(c != nullptr, "null context");
  CORR_CHECK_ARG(limit_ms >= 1 && limit_ms <= 2000,
                 "corr_selftest_wait_timeout: limit_ms must be in [1, 2000]");
  CORR_CUDA(cudaSetDevice(c->device));
  CORR_CUDA(cudaMemsetAsync(c->dres, 0, sizeof(ResultBlock), c->stream));
  wait_selftest_kernel<<<1, 32, 0, c->stream>>>((unsigned long long)limit_ms * 1000000ull,
                                                &c->dres->status);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  return finish_results(c, 0);
}

int corr_selftest_fp64(corr_context* c, int which, long long n, const double* x, double* out) {
  CORR_CHECK_ARG(c && x && out, "corr_selftest_fp64: null argument");
  CORR_CHECK_ARG(n >= 1 && (which == 0 || which == 1), "corr_selftest_fp64: bad n or function");
  CORR_CUDA(cudaSetDevice(c->device));
  CORR_TRY(c->ws.reserve((size_t)n * 16 + 512));
  Carver w{c->ws.ptr, 0};
  void* slot = w.take((size_t)n * 8);
  double* d_out = static_cast<double*>(w.take((size_t)n * 8));
  CORR_CUDA(cudaMemsetAsync(c->dres, 0, sizeof(ResultBlock), c->stream));
  const double* d_x = static_cast<const double*>(stage_in(c, x, (size_t)n * 8, slot));
  CORR_CHECK_ARG(d_x, "host-to-device copy failed");
  fp64_selftest_kernel<<<c->sms * 4, 256, 0, c->stream>>>(which, n, d_x, d_out);
  CORR_CUDA(cudaGetLastError());
  c->launches += 1;
  CORR_TRY(stage_out(c, out, d_out, (size_t)n * 8));
  return finish_results(c, 0);
}

int corr_selftest_factor(corr_context* c, int m, const double* J, double* L, double* X) {
  CORR_CHECK_ARG(c && J && L && X, "corr_selftest_factor: null argument");
  CORR_CHECK_ARG(m >= 1 && m <= 32768, "corr_selftest_factor: m must be in [1, 32768]");
  CORR_CUDA(cudaSetDevice(c->device));
  const size_t nj = (size_t)m * m * 8;
  auto plan = [&](Carver& w, void** p) {
    p[0] = w.take(nj);
    p[1] = w.take(nj);
    p[2] = w.take(nj);
    p[3] = w.take(chol_workspace_bytes(m));
    p[4] = w.take(dgemm_tc_workspace(m, m, m));
  };
  void* p[5];
  Carver cv{nullptr, 0};
  plan(cv, p);
  CORR_TRY(c->ws.reserve(cv.used));
  Carver w{c->ws.ptr, 0};
  plan(w, p);
  CORR_CUDA(cudaMemsetAsync(c->dres, 0, sizeof(ResultBlock), c->stream));
  const double* d_j = static_cast<const double*>(stage_in(c, J, nj, p[0]));
  CORR_CHECK_ARG(d_j, "host-to-device copy failed");
  double* d_x = static_cast<double*>(p[1]);
  double* d_l = nullptr;
  bool ok = false;
  CORR_TRY(chol_factor_inverse_device(c, p[3], d_j, m, 0.0, d_x, static_cast<double*>(p[2]), &d_l,
                                      &ok, p[4]));
  CORR_TRY(stage_out(c, L, d_l, nj));
  CORR_TRY(stage_out(c, X, d_x, nj));
  CORR_TRY(finish_results(c, 0));
  if (ok) return CORR_OK;
  set_error("corr_selftest_factor: a pivot is not positive and finite");
  return CORR_ERR_NOT_PD;
}

}  // extern "C"
