// Entry of the product for few rows and its fp16 instances (gemm_few.cuh).
#include "gemm_few.cuh"

// gemm_few_tcgen05.cu
int gemm_few_tcgen05(int wf, int dtype, const few::Operands& o, const few::Args& a, cudaStream_t st, bool pdl, int split);
int gemm_few_bf16(int wf, const few::Operands& o, const few::Args& a, cudaStream_t st, bool pdl, int split);

// out[M, N] = x . W^T (+ bias) (+ residual), or act(gate) * up with N / 2 columns, packed `w` of family `wf`, M <= 64 (32 with
// `pairs`: x then has 2 M rows, value and remainder of each token).  x: row stride ldx (a multiple of 8 elements), 16-byte
// aligned, as is w; K a multiple of 64.  split: CTAs that share a tile's k (1 .. 8; 0: chosen by the sizes).  -1: the
// driver refused a tensor map of the operands.
IPEX_API int ipex_gemm_few(const void* x, const void* w, void* out, const void* bias, const void* residual, const float* lut,
                           int M, int N, int K, int64_t ldx, int64_t ldo, int64_t ldr, int wf, int act, int pairs, int dtype,
                           int pdl, int split, int* err, void* stream) {
  const int rows = pairs ? 2 * M : M;
  if (M < 1 || rows > 64 || N < 1 || K < 1 || (K % 64) != 0 || (ldx % 8) != 0 || split < 0 || split > few::kMaxSplit)
    return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15)) return (int)cudaErrorInvalidValue;
  if (dtype != DT_F16 && dtype != DT_BF16) return (int)cudaErrorInvalidValue;
  if (act != 0 && (residual != nullptr || (N % 32) != 0)) return (int)cudaErrorInvalidValue;
  if (wf == WF_LUT4 && lut == nullptr) return (int)cudaErrorInvalidValue;
  if ((wf == WF_FP8_E4M3 || wf == WF_FP8_E5M2) && (K % 128) != 0) return (int)cudaErrorInvalidValue;
  const few::Operands o = {reinterpret_cast<const uint8_t*>(w), x, ldx, N, K};
  few::Args a = {};
  a.w = o.w; a.x = x; a.ldx = ldx; a.K = K;
  a.lut = lut;
  a.out = out; a.bias = bias; a.residual = residual; a.ldo = ldo; a.ldr = ldr;
  a.M = M; a.N = N;
  a.chunks = (K + 127) / 128;
  a.rows = rows;
  a.act = act;
  a.pairs = pairs;
  a.err = err;
  cudaStream_t st = (cudaStream_t)stream;
  // From 25 rows on (17 with minima) the weights' operand in tensor memory is the faster way (figures there); two rows to a token
  // keep the codes apart from their scales, which it does up to 32 columns or where a stage has one scale.
  const bool fp8 = wf == WF_FP8_E4M3 || wf == WF_FP8_E5M2;
  if (rows > (wf == WF_ASYM_INT4 ? 16 : 24) && (rows <= 32 || !pairs || fp8))
    return gemm_few_tcgen05(wf, dtype, o, a, st, pdl != 0, split);
  return dtype == DT_F16 ? few::by_family<__half>(wf, o, a, st, pdl != 0, split) : gemm_few_bf16(wf, o, a, st, pdl != 0, split);
}
