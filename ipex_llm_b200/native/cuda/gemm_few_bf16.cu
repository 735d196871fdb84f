// The bf16 instances of the product for few rows (gemm_few.cuh).
#include "gemm_few.cuh"

int gemm_few_bf16(int wf, const few::Operands& o, const few::Args& a, cudaStream_t st, bool pdl, int split) {
  return few::by_family<__nv_bfloat16>(wf, o, a, st, pdl, split);
}
