// spmm_f32.cu -- SpMM kernels instantiated for float B.
#include "spmm_impl.cuh"

namespace el {
EL_INSTANTIATE_SPMM(float)
}  // namespace el
