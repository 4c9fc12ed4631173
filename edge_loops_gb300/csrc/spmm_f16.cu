// spmm_f16.cu -- SpMM kernels instantiated for __half B.
#include "spmm_impl.cuh"

namespace el {
EL_INSTANTIATE_SPMM(__half)
}  // namespace el
