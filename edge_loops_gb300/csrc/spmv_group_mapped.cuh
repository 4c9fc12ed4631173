// spmv_group_mapped.cuh -- the reference's group_mapped schedule
// [include/loops/schedule/group_mapped.hxx:146-235,
// include/loops/algorithms/spmv/group_mapped.cuh:26-60]: a group of GT threads
// (GT = 32 is the reference's warp_mapped, GT = block size its block_mapped)
// owns GT consecutive rows and shares their nonzeros among its threads.  Here
// each warp of the group takes 32 of its rows (or, when there are groups
// enough for that, a warp the whole group) and walks their nonzeros in tiles of
// 256 with the merge-path walk, whose lanes own consecutive nonzeros and find
// the row ends among them by bits instead of an upper bound per nonzero.
// Whole rows per warp: no carries, no barrier.
//
// One nonzero per thread and chunk, a block scan and two barriers per 128
// nonzeros took 188 us on a 96^3 stencil (23.4M nonzeros, FP32).
#pragma once

#include "spmv_merge_path_nz.cuh"

namespace el {
namespace mpn {

template <typename VT, bool COMP>
__global__ void __launch_bounds__(kTPB, 3)
    group_mapped_kernel(const Src m, WsHeader* hdr, const int rows_per_warp) {
  __shared__ WarpSmem<COMP> smem[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long step = (long long)gridDim.x * kWarps * rows_per_warp;
  bool bad = false, bad_col = false;
  auto bound = [&](long long r) { return __ldg(m.offsets + min(r, (long long)m.rows)); };
  long long r0 = ((long long)blockIdx.x * kWarps + warp) * rows_per_warp;
  int b = bound(r0), e = bound(r0 + rows_per_warp);
  for (; r0 < m.rows; r0 += step) {  // warp-uniform
    // the next rows' bounds are in flight during the walk
    const int nb = bound(r0 + step), ne = bound(r0 + step + rows_per_warp);
    bad |= b < 0 || e < b || e > m.nnz;
    const int lo = min(max(b, 0), m.nnz), hi = min(max(e, lo), m.nnz);
    const int r1 = (int)min(r0 + rows_per_warp, (long long)m.rows);
    int ra = (int)r0;
    (void)walk_rows<VT, COMP>(m, smem[warp], lane, (int)r0, r1, lo, hi, false, bad, bad_col, ra);
    bad |= ra < r1;
    b = nb;
    e = ne;
  }
  if (__any_sync(kFullMask, bad_col) && lane == 0) raise_flag(hdr, EL_FLAG_INDEX_RANGE, 0);
  if (__any_sync(kFullMask, bad) && lane == 0) raise_flag(hdr, EL_FLAG_OFFSETS, 0);
}

template <typename VT, bool COMP>
el_status launch_group_mapped_rows(const SpmvCall& c, int group_rows) {
  const int per_sm = resident_ctas_per_sm((const void*)group_mapped_kernel<VT, COMP>, kTPB, 0, true);
  const long long ctas = (long long)(per_sm > 0 ? per_sm : 1) * device_info(c.device).sm_count;
  Src m{c.A.offsets, c.A.indices, c.A.values, c.A.row_scale, c.x, c.y,
        (int)c.A.rows, (unsigned)c.A.cols, (int)c.A.nnz, 0, 0};
  tile_phase(c.A.indices, c.A.values, (int)sizeof(VT), &m.vec_ok, &m.ph);
  // A warp takes the whole group (four together where a group is 32 rows)
  // where that leaves 1.5 chunks per resident warp, else fewer rows, down to
  // 32: whole tiles against warps left idle.
  // 32 / 64 / 128 rows per warp: stencil 96^3 (885k rows) 76 / 64 / 60 us,
  // 2M log-normal rows of 8 117 / 101 / 91, stencil 40^3 (64k rows) 15 / 17 /
  // 25, 100k uniform rows of 35 25 / 29 / 31 (a block scan per 128 nonzeros:
  // 191, 156, 29, 48).
  int rpw = group_rows > 128 ? group_rows : 128;
  while (rpw > 32 && c.A.rows * 2 < 3 * ctas * kWarps * rpw) rpw /= 2;
  const long long chunks = (c.A.rows + rpw - 1) / rpw;
  long long grid = (chunks + kWarps - 1) / kWarps;
  if (grid > ctas) grid = ctas;
  group_mapped_kernel<VT, COMP><<<(unsigned)grid, kTPB, 0, c.stream>>>(m, c.ws.hdr, rpw);
  return cuda_status(cudaGetLastError(), "group_mapped launch");
}

}  // namespace mpn
}  // namespace el
