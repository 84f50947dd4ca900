// tag_eval_means: evaluates device forms of the logarithmic and Stolarsky means
// (kinds 0, 3, 4, 7 and 8 the kernels' own inline functions, the others FP64 forms
// to hold them against) on arrays of value pairs, so that they can be checked
// directly against exact values on both sides of every branch threshold.  Diagnostics only: no kernel of the right-hand side calls
// this path.
#include <cuda_runtime.h>

#include <string>

#include "phys_pt_2d.cuh"
#include "tag_common.cuh"

using namespace tag;

namespace {

int mfail(int code, const std::string& msg) {
  set_last_error(msg);
  return code;
}

// kind 0: the element kernels' integer forms from node logarithms (ln_factor,
//         and inv_ln_factor of the reciprocals); kind 3: the interface kernels'
//         forms of the values themselves
// kinds 1, 2: the FP64 polynomial forms of halved values with per-node
//         logarithms, ranges 0.01 (1) and 0.09 (2)
// kind 4: Stolarsky mean of the potential-temperature kernels (out2 unused)
// kind 5: as kind 2 with the pair as the ln_mean pair and (1, 1) as the
//         inv_ln_mean pair; kind 6 the other way round
// out1 = ln_mean(x, y) (kind 4: the Stolarsky mean), out2 = inv_ln_mean(x, y);
// kinds 5 and 6 return the means of their (x, y) and (1, 1) pairs.
// kind 7: int_rcp(x) and int_rsqrt(y); kind 8: int_pow(x, gamma) and int_exp(y)
__global__ void k_eval_means(int kind, long n, const double* __restrict__ x,
                             const double* __restrict__ y, PhysPT2D::Params pt,
                             double* __restrict__ out1, double* __restrict__ out2) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double a = x[q], b = y[q];
  double m = 0.0, im = 0.0;
  if (kind == 0) {
    const double ia = int_rcp(a), ib = int_rcp(b);
    m = 0.5 * (a + b) * ln_factor(a, b, log_difference(log_word(a), log_word(b)));
    im = 0.5 * (ia + ib) * inv_ln_factor(ia, ib, log_difference(log_word(ia), log_word(ib)));
  } else if (kind == 1 || kind == 2) {
    const double ha = 0.5 * a, hb = 0.5 * b;
    const double la = log(ha), lb = log(hb);
    if (kind == 1)
      ln_mean_pair_halved<true, false>(ha, hb, ha, hb, la, lb, la, lb, m, im);
    else
      ln_mean_pair_halved(ha, hb, ha, hb, la, lb, la, lb, m, im);
  } else if (kind == 5 || kind == 6) {
    const double ha = 0.5 * a, hb = 0.5 * b;
    const double la = log(ha), lb = log(hb), l1 = log(0.5);
    if (kind == 5)
      ln_mean_pair_halved(ha, hb, 0.5, 0.5, la, lb, l1, l1, m, im);
    else
      ln_mean_pair_halved(0.5, 0.5, ha, hb, l1, l1, la, lb, m, im);
  } else if (kind == 3) {
    m = ln_mean_of(a, b);
    im = inv_ln_mean_of_reciprocals(int_rcp(a), int_rcp(b));
  } else if (kind == 7) {
    m = int_rcp(a);
    im = int_rsqrt(b);
  } else if (kind == 8) {
    m = int_pow(a, pt.gamma, pt.gamma_q61);
    im = int_exp(b);
  } else {
    m = PhysPT2D::stolarsky(pt, a, b);
  }
  out1[q] = m;
  out2[q] = im;
}

}  // namespace

extern "C" {

int tag_eval_means(int32_t kind, int64_t n, double gamma_cp, double gamma_cv, const double* x,
                   const double* y, double* out1, double* out2) {
  if (kind < 0 || kind > 8 || n < 0 || (n > 0 && (!x || !y || !out1 || !out2)))
    return mfail(TAG_E_INVALID, "tag_eval_means: bad argument");
  if (n == 0) return TAG_OK;
  const double pp[8] = {gamma_cp, gamma_cv, 9.81, 340.0, 0.0, 0.0, 0.0, 1.0};
  const PhysPT2D::Params pt = PhysPT2D::make_params(pp);
  double* d = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  cudaError_t e = cudaMalloc(&d, 4 * bytes);
  if (e != cudaSuccess) return mfail(TAG_E_CUDA, cudaGetErrorString(e));
  e = cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, y, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_eval_means<<<(unsigned)((n + 255) / 256), 256>>>(kind, n, d, d + n, pt, d + 2 * n, d + 3 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out1, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(out2, d + 3 * n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return mfail(TAG_E_CUDA, cudaGetErrorString(e));
  return TAG_OK;
}

}  // extern "C"
