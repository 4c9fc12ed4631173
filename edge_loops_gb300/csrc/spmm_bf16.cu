// spmm_bf16.cu -- SpMM kernels instantiated for __nv_bfloat16 B.
#include "spmm_impl.cuh"

namespace el {
EL_INSTANTIATE_SPMM(__nv_bfloat16)
}  // namespace el
