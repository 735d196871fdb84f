// One entry for a packed linear layer on few rows: which kernel takes them is decided here, in one call, because at this size
// the host's work is longer than the GPU's (one row of 4096 x 4096: 6.6 us of kernel).
#include "common/utils.cuh"

IPEX_API int ipex_gemm_few(const void* x, const void* w, void* out, const void* bias, const void* residual, const float* lut,
                           int M, int N, int K, int64_t ldx, int64_t ldo, int64_t ldr, int wf, int act, int pairs, int dtype,
                           int pdl, int split, int* err, void* stream);
IPEX_API int ipex_gemv_lowbit_stream(const void* w, int wf, const void* x, void* y, int M, int N, int K, int ldx, int ldy,
                                     const void* norm_w, float eps, float norm_offset, const void* bias, const void* residual,
                                     int ldr, int act, const float* lut, int dtype, int pdl, int* err, void* stream);

// out[M, N] = x[M, K] . W^T, rows one after another in 16 bits, packed `w` of family `wf`.  faster: the product for few rows
// is the faster one for these rows and loses no precision against the GEMVs (for more than eight rows: always).  Returns
// cudaErrorInvalidValue, and launches nothing, for what these kernels do not take; the general way is the caller's then.
IPEX_API int ipex_linear_rows(const void* x, const void* w, void* out, const float* lut, int M, int N, int K, int wf, int dtype,
                              int faster, int* err, void* stream) {
  if (faster) return ipex_gemm_few(x, w, out, nullptr, nullptr, lut, M, N, K, K, N, 0, wf, 0, 0, dtype, 0, 0, err, stream);
  if (wf != WF_SYM_INT4 && wf != WF_FP8_E4M3) return (int)cudaErrorInvalidValue;
  return ipex_gemv_lowbit_stream(w, wf, x, out, M, N, K, K, N, nullptr, 0.f, 0.f, nullptr, nullptr, 0, 0, nullptr, dtype, 0, err,
                                 stream);
}
