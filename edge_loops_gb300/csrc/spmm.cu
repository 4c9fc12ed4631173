// spmm.cu -- dispatch of the SpMM launchers (spmm_impl.cuh) by type, and the
// workspace they need.
#include "el_internal.h"

namespace el {

// Warp ranges of the merge-path SpMM, at most: 48 per SM (24 are resident),
// with a carry slot and a row vector of 128 floats each.  No more slots than a
// new workspace has: one that grew would leave a graph captured before with
// the memory it had.
static long long spmm_mp_ranges(const SpmmCall& c) {
  return (long long)device_info(c.device).sm_count * 48;
}

size_t spmm_scratch_bytes(const SpmmCall& c, int schedule) {
  if (schedule != EL_SCHED_MERGE_PATH_FLAT) return 0;
  return (size_t)spmm_mp_ranges(c) * 128 * sizeof(float);
}

long long spmm_slots_needed(const SpmmCall& c, int schedule) {
  return schedule == EL_SCHED_MERGE_PATH_FLAT ? spmm_mp_ranges(c) : 0;
}

el_status launch_spmm(const SpmmCall& c, int schedule) {
  const int vt = c.A.value_dtype, bt = c.b_dtype;
  if ((vt == EL_BF16 && bt == EL_F16) || (vt == EL_F16 && bt == EL_BF16))
    return fail(EL_ERR_UNSUPPORTED, "SpMM value/B dtype pair (%d, %d) not built", vt, bt);
  switch (bt) {
    case EL_F32: return spmm_launch<float>(c, schedule);
    case EL_BF16: return spmm_launch<__nv_bfloat16>(c, schedule);
    default: return spmm_launch<__half>(c, schedule);
  }
}

}  // namespace el
