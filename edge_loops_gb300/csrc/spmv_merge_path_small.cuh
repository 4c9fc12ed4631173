// spmv_merge_path_small.cuh -- the merge-path SpMV for small matrices.
//
// Same split as spmv_merge_path_nz.cuh (equal merge ranges at diagonals
// g * range_items, the reference's search [include/loops/schedule/
// merge_path_flat.hxx:108-138, util/search.hxx:34-60]), but a range is a
// CTA's: with everything resident at once the time is a chain of memory round
// trips, so the CTA makes few of them -- offsets (all of them when there are
// few rows, while the ticket is on its way), columns and values, x -- puts
// the products in shared memory and sums rows from there, L lanes per row by
// the range's mean row length.  A row begun shortly before the range is
// multiplied again from its start instead of waiting for the earlier range's
// partial.
#pragma once

#include "spmv_merge_path_nz.cuh"

namespace el {
namespace mpn {

constexpr int kSmTPB = 256;
constexpr int kSmItems = 2048;    // merge items per range, at most
constexpr int kSmRows = 4096;     // rows whose offsets a CTA holds, at most
constexpr int kSmAgain = 1024;    // nonzeros of an earlier range multiplied again, at most
constexpr int kSmLong = 8;        // rows longer than this many per lane: a warp each
constexpr int kSmLongRows = (kSmItems + kSmAgain) / (kSmLong + 1) + 1;

struct SmallSmem {
  float prod[kSmItems + kSmAgain];
  int off[kSmRows + 2];  // offsets of the range's rows (or of all rows)
  int long_rows[kSmLongRows];
  int n_long;
  unsigned ticket[2];
  SplitPoint sp[2];
};

template <typename VT>
__global__ void __launch_bounds__(kSmTPB) merge_path_small_kernel(const Args a) {
  __shared__ SmallSmem S;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  WsHeader* const hdr = a.ws.hdr;
  const float* __restrict__ scale = a.row_scale;
  const bool few = a.rows <= kSmRows;  // every offset fits
  if (t == 0) {
    S.n_long = 0;
    take_ticket(hdr, gridDim.x, &S.ticket[0], &S.ticket[1]);
  }
  if (few)
    for (int i = t; i <= (int)a.rows; i += kSmTPB) S.off[i] = __ldg(a.offsets + i);
  __syncthreads();
  const long long g = S.ticket[0];
  const unsigned tag = epoch_tag(S.ticket[1]);
  const long long w = a.rw, total = w * a.rows + a.nnz;
  const long long d0 = min(g * a.range_items, total), d1 = min(d0 + a.range_items, total);
  SplitPoint sa, sb;
  if (few) {
    warp_merge_search2_w([&](long long k) { return S.off[k + 1]; }, a.rows, a.nnz, d0, d1, w, sa,
                         sb);
  } else {
    if (warp == 0) {
      warp_merge_search2_w([&](long long k) { return __ldg(a.offsets + 1 + k); }, a.rows, a.nnz,
                           d0, d1, w, sa, sb);
      if (lane == 0) {
        S.sp[0] = sa;
        S.sp[1] = sb;
      }
    }
    __syncthreads();
    sa = S.sp[0];
    sb = S.sp[1];
  }
  const int rs = (int)sa.x, re = (int)sb.x;
  const int ns = split_nonzero(sa, d0, w, a.rows);
  const int ne = split_nonzero(sb, d1, w, a.rows);
  if (a.trace && g < a.trace_cap && t < 6) {
    const long long t6[6] = {d0, d1, rs, ns, re, ne};
    long long tv = t6[0];
#pragma unroll
    for (int k = 1; k < 6; ++k)
      if (t == k) tv = t6[k];
    a.trace[6 * g + t] = tv;
  }
  if (t == 0) {
    if (g == 0 && sa.start != 0) raise_flag(hdr, EL_FLAG_NNZ_MISMATCH, 0);
    if (re == (int)a.rows && sb.start != (int)a.nnz)
      raise_flag(hdr, EL_FLAG_NNZ_MISMATCH, (unsigned)re);
  }
  // row rs began before the range: again from its start, or by the look-back
  const bool inside = ns > sa.start && rs < re;
  const bool again = inside && sa.start >= 0 && ns - sa.start <= kSmAgain;
  const int n0 = again ? sa.start : ns;
  const int len = min(ne - n0, kSmItems + kSmAgain);  // (never cut on well-formed offsets)

  // products
  const VT* __restrict__ vals = reinterpret_cast<const VT*>(a.values);
  bool bad = false;
  for (int k0 = t; k0 < len; k0 += 4 * kSmTPB) {
    int c[4];
    float v[4], xv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + u * kSmTPB;
      c[u] = k < len ? __ldcs(a.indices + n0 + k) : 0;
      v[u] = k < len ? to_f32(vals[n0 + k]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // a column outside [0, cols) adds 0 and reads nothing
      const bool in = k0 + u * kSmTPB < len;
      const bool ok = (unsigned)c[u] < (unsigned long long)a.cols;
      bad |= in && !ok;
      xv[u] = in && ok ? __ldg(a.x + c[u]) : 0.f;
      if (!ok) v[u] = 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k0 + u * kSmTPB < len) S.prod[k0 + u * kSmTPB] = __fmul_rn(v[u], xv[u]);
  }
  if (bad) raise_flag(hdr, EL_FLAG_INDEX_RANGE, (unsigned)rs);
  const int ob = few ? rs : 0;  // off[ob + i]: start of row rs + i
  int nr = re - rs;
  if (nr < 0 || (!few && nr > kSmRows)) {  // malformed offsets
    raise_flag(hdr, EL_FLAG_OFFSETS, (unsigned)rs);
    nr = nr < 0 ? 0 : kSmRows;
  }
  if (!few)
    for (int i = t; i <= nr; i += kSmTPB) S.off[i] = __ldg(a.offsets + rs + i);
  __syncthreads();

  // sum of products [b, e) by the warp: four sums per lane, then their tree
  // (short chains, for the rounding error as for the time)
  auto warp_sum = [&](int b, int e) {
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = b + lane; k < e; k += 128) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + 32 * u < e) s4[u] = __fadd_rn(s4[u], S.prod[k + 32 * u]);
    }
    float s = __fadd_rn(__fadd_rn(s4[0], s4[1]), __fadd_rn(s4[2], s4[3]));
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s = __fadd_rn(s, __shfl_xor_sync(kFullMask, s, d));
    return s;
  };
  // the row left open: its partial goes to the range where it ends
  if (warp == kSmTPB / 32 - 1) {
    const int lo = max(sb.start, ns);
    if (ne > lo) {
      const float s = warp_sum(min(lo - n0, len), len);
      if (lane == 0 && g < a.ws.nslots && !(a.test_hooks & 1)) {
        publish_carry<false>(a.ws.slots + g, s, 0.f, tag);
      }
    }
  }
  // rows: L lanes each, by the mean length; long ones and row rs, when it
  // waits for earlier ranges, by a warp each
  const int mean = nr > 0 ? len / nr : 0;
  const int L = mean < 3 ? 1 : mean < 6 ? 2 : mean < 12 ? 4 : mean < 24 ? 8 : mean < 48 ? 16 : 32;
  const int sub = t & (L - 1);
  for (int i0 = 0; i0 < nr; i0 += kSmTPB / L) {  // CTA-uniform
    const int i = i0 + t / L;
    float s = 0.f;
    bool mine = i < nr;
    if (mine) {
      int b = S.off[ob + i] - n0, e = S.off[ob + i + 1] - n0;
      if (e < b || e > len || (b < 0 && i > 0)) {
        raise_flag(hdr, EL_FLAG_OFFSETS, (unsigned)(rs + i));
        e = min(max(e, 0), len);
      }
      b = min(max(b, 0), e);
      if (e - b > kSmLong * L || (i == 0 && inside && !again)) {
        mine = false;
        if (sub == 0) {
          const int q = atomicAdd(&S.n_long, 1);
          if (q < kSmLongRows) S.long_rows[q] = i;
        }
      } else {
        for (int k = b + sub; k < e; k += L) s = __fadd_rn(s, S.prod[k]);
      }
    }
    for (int d = L >> 1; d > 0; d >>= 1) s = __fadd_rn(s, __shfl_xor_sync(kFullMask, s, d));
    if (mine && sub == 0) a.y[rs + i] = scale ? s * __ldg(scale + rs + i) : s;
  }
  __syncthreads();
  const int nl = min(S.n_long, kSmLongRows);
  for (int q = warp; q < nl; q += kSmTPB / 32) {
    const int i = S.long_rows[q];
    const int e = min(max(S.off[ob + i + 1] - n0, 0), len);
    float s = warp_sum(min(max(S.off[ob + i] - n0, 0), e), e);
    if (i == 0 && inside && !again) {
      bool ok;
      Acc<false> acc = look_back<false>(a, (w * rs + sa.start) / a.range_items, g, tag, ok);
      if (!ok && lane == 0) raise_flag(hdr, EL_FLAG_TIMEOUT, 4);
      s = __fadd_rn(acc.s, s);
    }
    if (lane == 0) a.y[rs + i] = scale ? s * __ldg(scale + rs + i) : s;
  }
}

// Four ranges of 2048 items per SM at most (five CTAs are resident), and no
// option that shapes the warp walk.  Passes after each other on the GB300, this
// kernel / the warp walk, log-normal rows of 13: 20,000 nonzeros 8.2 / 10.5 us,
// 60,000 8.2 / 12.3, 200,000 10.3 / 12.4, 300,000 10.3 / 12.4, 500,000 12.3 /
// 14.4, 800,000 14.4 / 16.4, 1.2M 16.5 / 18.6, 1.6M 18.5 / 18.6, 4M 39 / 29
// (from there on the walk's 24 warps per SM hide more than the shorter chain
// saves).
constexpr int kSmCtasPerSm = 4;
template <typename VT>
bool small_fits(const SpmvCall& c) {
  if (c.o.max_ctas > 0 || c.o.nz_per_lane != 0) return false;
  const long long total = (long long)row_weight(c) * c.A.rows + c.A.nnz;
  return total <= (long long)device_info(c.device).sm_count * kSmCtasPerSm * kSmItems;
}

template <typename VT>
el_status launch_small(const SpmvCall& c) {
  Args a;
  a.rw = row_weight(c);
  const long long total = (long long)a.rw * c.A.rows + c.A.nnz;
  // whole 256-item units, as the warp ranges; four CTAs per SM cover each
  // other's round trips (300,000 nonzeros: 12.3 us in ranges of 2048, 10.3 of
  // 1024; 1.2M: 16.5 of 2048, 20.3 of 1024, two waves)
  const long long ctas = (long long)device_info(c.device).sm_count * kSmCtasPerSm;
  const long long units = (total + kTileNz - 1) / kTileNz, upr = (units + ctas - 1) / ctas;
  a.rows = c.A.rows;
  a.cols = c.A.cols;
  a.nnz = c.A.nnz;
  a.offsets = c.A.offsets;
  a.indices = c.A.indices;
  a.values = c.A.values;
  a.row_scale = c.A.row_scale;
  a.x = c.x;
  a.y = c.y;
  a.range_items = upr * kTileNz;
  a.num_ranges = (units + upr - 1) / upr;
  a.vec_ok = a.ph = 0;
  a.test_hooks = c.o.test_hooks;
  a.wait_ns = c.wait_ns;
  a.ws = c.ws;
  a.trace = c.trace;
  a.trace_cap = c.trace_cap;
  if (a.num_ranges > c.ws.nslots)
    return fail(EL_ERR_INVALID_ARGUMENT, "merge_path: workspace too small");
  merge_path_small_kernel<VT><<<(unsigned)a.num_ranges, kSmTPB, 0, c.stream>>>(a);
  return cuda_status(cudaGetLastError(), "merge_path launch");
}

}  // namespace mpn
}  // namespace el
