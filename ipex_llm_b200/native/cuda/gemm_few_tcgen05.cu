// The instances of gemm_few_tcgen05.cuh.
#include "gemm_few_tcgen05.cuh"

template <typename T>
static int any_family(int wf, const few::Operands& o, const few::Args& a, cudaStream_t st, bool pdl, int split) {
  using namespace few::tm;
  switch (wf) {
    case WF_SYM_INT4: return by_width<T, WF_SYM_INT4>(o, a, st, pdl, split);
    case WF_ASYM_INT4: return by_width<T, WF_ASYM_INT4>(o, a, st, pdl, split);
    case WF_LUT4: return by_width<T, WF_LUT4>(o, a, st, pdl, split);
    case WF_FP8_E4M3: return by_width<T, WF_FP8_E4M3>(o, a, st, pdl, split);
    case WF_FP8_E5M2: return by_width<T, WF_FP8_E5M2>(o, a, st, pdl, split);
    case WF_INT8: return by_width<T, WF_INT8>(o, a, st, pdl, split);
    default: return (int)cudaErrorInvalidValue;
  }
}

int gemm_few_tcgen05(int wf, int dtype, const few::Operands& o, const few::Args& a, cudaStream_t st, bool pdl, int split) {
  return dtype == DT_F16 ? any_family<__half>(wf, o, a, st, pdl, split) : any_family<__nv_bfloat16>(wf, o, a, st, pdl, split);
}
