// spmm_impl.cuh -- CSR SpMM C = A B for sm_103a (B, C dense row-major),
// included once per B type (spmm_f32.cu, spmm_bf16.cu, spmm_f16.cu).
//
// One kernel runs the three schedules.  The nonzeros are cut into equal
// warp ranges along the merge path of row ends and nonzeros, and a warp's
// range into one PIECE per group of G lanes (G = 4 .. 32, by the width of a
// B row), so a warp walks 32 / G pieces in step, U nonzeros of each at a
// time, with the B reads of a step in flight together.  The reads of B are
// random; what bounds the walk is how many of them the resident warps keep
// in flight and the instructions between them, so a step waits on nothing
// else: its columns and values are loaded a step ahead, and the row ends of
// the range are read once, before the walk, into a bit per nonzero in shared
// memory.
//
//  merge_path: ranges and pieces are cut anywhere; rows that cross pieces
//    are stitched in shared memory, rows that cross ranges by row-vector
//    carries that the range where the row ends collects (range ids from an
//    atomic ticket, bounded spins, fixed order: deterministic).
//  thread_mapped, group_mapped (ORDERED): cuts are moved to row starts, and
//    every C element is summed in nonzero order without fused multiply-add,
//    the reference's order [algorithms/spmm/thread_mapped.cuh:28-53]: equal
//    bit for bit to the CPU loop.
// At most 128 columns per pass; wider B is processed in column blocks.
#pragma once

#include "el_internal.h"

namespace el {
namespace spmm {

constexpr int kPassCols = 128;  // columns per pass, at most
constexpr int kWarps = 4;       // per CTA
constexpr int kTPB = 32 * kWarps;
constexpr int kBlock = 4096;    // merge items of a range worked on at a time
constexpr int kMaxNz = 2 * kBlock;  // nonzeros of a block, at most
constexpr int kFold = 32;           // steps (a power of two)
// ORDERED: longer rows are walked by the whole warp, which has 32 / G times the
// B rows in flight (a group alone takes 0.45 us per 8 nonzeros); shorter ones
// cost more to set apart than that saves.  Threshold none / 512 / 256 / 128:
// 3,000 log-normal rows of 20, n = 9, 74 / 44 / 35 / 31 us; 60,000 of them,
// n = 64, 93 / 70 / 64 / 64; 200,003 of 10, n = 24, 58 / 58 / 58 / 70.
// Ranges of fewer items set shorter rows apart (launch_kernel): one row is
// most of a warp's time there.  30,000 nonzeros in log-normal rows of 4, n = 4:
// 32 us at 256, 17 at 64, 16 at 32; 300,000 in rows of 38: 20.0 / 20.0 / 17.9.
constexpr int kLongRow = 256;
// Merge items per row end: a row end costs the walk about two nonzeros (its
// test, store and new sum).
constexpr int kRowItems = 2;
constexpr int kMaxRows = kBlock / kRowItems + 1;  // rows of a block, at most
// Resident CTAs per SM: 24 warps of 80 registers (8M nonzeros, n = 32: 187 µs;
// 20 warps of 96: 205; 32 of 64, which spills in the walk: 230).
constexpr int kMinCtas = 6;

struct Args {
  long long rows, cols, nnz;
  const int* offsets;
  const int* indices;
  const unsigned char* values;
  int value_dtype;
  const float* row_scale;
  const unsigned char* B;      // the whole B
  unsigned long long ldb;      // bytes from one row of B to the next
  unsigned long long b_first;  // bytes from a row's start to this pass's first column
  float* C;                    // this pass's first column
  long long ldc;
  int n;  // columns in this pass
  long long range_items;  // merge items per warp
  int block_items;        // of them worked on at a time, at most kBlock
  int long_row;           // ORDERED, several groups per warp: rows set apart from here on
  long long num_ranges;
  WsHeader* hdr;
  CarrySlot* flags;
  float* vec;  // num_ranges x kPassCols row-vector carries
  unsigned long long wait_ns;
  int test_hooks;
};

// --------------------------------------------------------------- B elements
template <typename BT>
__device__ __forceinline__ float bits_to_f32(uint32_t h);
template <>
__device__ __forceinline__ float bits_to_f32<float>(uint32_t h) {
  return __uint_as_float(h);
}
template <>
__device__ __forceinline__ float bits_to_f32<__nv_bfloat16>(uint32_t h) {
  return __uint_as_float(h << 16);
}
template <>
__device__ __forceinline__ float bits_to_f32<__half>(uint32_t h) {
  return __half2float(__ushort_as_half((unsigned short)h));
}

// How a group of G lanes holds a B row: K blocks of V adjacent columns per
// lane (V elements are one load: rows of B and C start on such boundaries and
// n is whole vectors; V = 1 takes any alignment and width).
template <typename BT, int V_, int K_, int G_>
struct Lay {
  using T = BT;
  static constexpr int V = V_, K = K_, G = G_;
  static constexpr int P = V * K;                           // columns per lane
  static constexpr int kCols = G * P;                       // columns per group
  static constexpr int kWords = (V * (int)sizeof(BT) + 3) / 4;  // registers per load
  static constexpr int U = G < 8 ? G : 8;                   // nonzeros per step
  static __device__ __forceinline__ int column(int sl, int k) { return V * (sl + G * k); }
};

// V adjacent elements of a B row, as loaded.
template <typename L>
struct BVec {
  using BT = typename L::T;
  uint32_t w[L::kWords];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < L::kWords; ++i) w[i] = 0u;
  }
  __device__ __forceinline__ void load(const unsigned char* p) {
    constexpr int kB = L::V * (int)sizeof(BT);
    if constexpr (kB == 16) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
      w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
    } else if constexpr (kB == 8) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
      w[0] = u.x; w[1] = u.y;
    } else if constexpr (kB == 4) {
      w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
    } else {
      w[0] = __ldg(reinterpret_cast<const unsigned short*>(p));
    }
  }
  __device__ __forceinline__ float get(int i) const {
    if (sizeof(BT) == 4) return __uint_as_float(w[i]);
    return bits_to_f32<BT>((i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu);
  }
};

// A nonzero as loaded (nothing waits on the loads before use).
struct Nz {
  int c;
  uint32_t v;  // the value's bits
  __device__ __forceinline__ void load(const Args& a, bool in, unsigned at) {
    c = -1;
    v = 0u;
    if (in) {
      c = __ldcs(a.indices + at);
      if (a.value_dtype == EL_F32)
        v = __ldcs(reinterpret_cast<const uint32_t*>(a.values) + at);
      else
        v = __ldcs(reinterpret_cast<const unsigned short*>(a.values) + at);
    }
  }
  __device__ __forceinline__ float value(const Args& a) const {
    return a.value_dtype == EL_F32    ? __uint_as_float(v)
           : a.value_dtype == EL_BF16 ? bits_to_f32<__nv_bfloat16>(v)
                                      : bits_to_f32<__half>(v);
  }
};

template <typename L, bool ORDERED>
struct Smem {  // per warp
  static constexpr int NG = 32 / L::G;
  __align__(16) int idx[2][32];    // a step's columns (-1: none)
  __align__(16) float val[2][32];  // and values
  float sc[2][32];                 // scales of the G rows from the step's first on
  unsigned ends[kMaxNz / 32 + 4];  // bit i: a row ends after the block's nonzero i
  unsigned rowm[kMaxRows / 32 + 4];  // bit i: row i of the block ends by such a bit
  float open[ORDERED ? 1 : NG][ORDERED ? 1 : L::kCols];  // a piece's open row
  float pend[ORDERED ? 1 : NG][ORDERED ? 1 : L::kCols];  // its part of the row it began inside
  float fold[ORDERED ? 1 : L::P][32];  // the lanes' earlier sums of a long row
  int first[NG];     // a piece's first row
  int closed[NG];    // it closed a row
  int has_pend[NG];  // that first row began before the piece
};

// bits [at, at + 32) of a bit array
__device__ __forceinline__ unsigned bits_at(const unsigned* m, int at) {
  return __funnelshift_r(m[at >> 5], m[(at >> 5) + 1], at & 31);
}

struct RowSmem {  // per warp, where it takes whole rows
  int idx[2][32];
  float val[2][32];
};

template <typename L, bool ORDERED, typename Sm_ = Smem<L, ORDERED>>
struct Walk {
  using Sm = Sm_;
  static constexpr int G = L::G, U = L::U, NG = 32 / G, P = L::P, V = L::V, K = L::K;
  // (a block closes at most kBlock nonzeros beside its first row's)
  const Args& a;
  Sm& M;
  const int lane, sl, grp;
  bool bad_col = false, bad_off = false;
  const unsigned char* my_B[K];  // the lane's columns of row 0 of B

  __device__ __forceinline__ Walk(const Args& a_, Sm& m_)
      : a(a_), M(m_), lane(threadIdx.x & 31), sl(lane & (G - 1)), grp(lane / G) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = L::column(sl, k);  // past the last column: reads the first again
      my_B[k] = a.B + a.b_first + (c < a.n ? c : 0) * sizeof(typename L::T);
    }
  }

  static __device__ __forceinline__ float mad(float v, float b, float acc) {
    return ORDERED ? __fadd_rn(acc, __fmul_rn(v, b)) : __fmaf_rn(v, b, acc);
  }
  static __device__ __forceinline__ void add(float v, const BVec<L> (&b)[K], float (&acc)[P]) {
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[V * k + i] = mad(v, b[k].get(i), acc[V * k + i]);
  }

  // acc -> the C row whose lane's first column is at dst (streamed: C is not
  // read again)
  __device__ __forceinline__ void store(float* dst, const float (&acc)[P], float s) const {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (L::column(sl, k) >= a.n) continue;
      float* const d = dst + V * G * k;
      const float* const t = acc + V * k;
      if constexpr (V == 1)
        __stcs(d, t[0] * s);
      else if constexpr (V == 2)
        __stcs(reinterpret_cast<float2*>(d), make_float2(t[0] * s, t[1] * s));
      else
#pragma unroll
        for (int i = 0; i < V; i += 4)
          __stcs(reinterpret_cast<float4*>(d + i),
                 make_float4(t[i] * s, t[i + 1] * s, t[i + 2] * s, t[i + 3] * s));
    }
  }

  // The sums of one step: every row end is a store under a predicate.  GAP:
  // rows skip the empty ones (rw: the rows from the current one on as bits);
  // SC: rows are scaled.
  template <bool GAP, bool SC>
  __device__ __forceinline__ void sums(const BVec<L> (&b)[U][K], const float (&v)[U],
                                       unsigned ends, unsigned rw, const float* sc,
                                       float (&acc)[P], float*& crow) const {
    int moved = 0;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      add(v[j], b[j], acc);
      if ((ends >> j) & 1u) {
        store(crow, acc, SC ? sc[moved] : 1.f);
        int gap = 1;
        if (GAP) {
          gap = __ffs(rw >> 1);
          rw >>= gap;
        }
        crow += GAP ? gap * a.ldc : a.ldc;
        if (SC) moved += gap;
#pragma unroll
        for (int k = 0; k < P; ++k) acc[k] = 0.f;
      }
    }
  }

  // One row, nonzeros [b, e) in order, by the whole warp: the groups read
  // the B rows of NG U nonzeros at once and add their products in turn, each
  // group to the sum the one before it hands on.
  // LEAN: the shorter code, for the walk, which it slows less (166,000 log-normal
  // rows of 12, n = 16: 65 us lean, 78 not; a warp per row, BF16 B, n = 33, 5,000
  // of them: 53 us lean, 27 not).
  template <bool LEAN>
  __device__ __forceinline__ void whole_row(int row, int b, int e) {
    float acc[P];
#pragma unroll
    for (int k = 0; k < P; ++k) acc[k] = 0.f;
    Nz nz;
    const int mine = grp * U + sl;  // this lane's nonzero of a step (sl < U)
    nz.load(a, sl < U && b + mine < e, b + mine);
    int slot = 0;
#pragma unroll 1
    for (int y = b; y < e; y += NG * U, slot ^= 1) {
      const bool ok = (unsigned)nz.c < (unsigned long long)a.cols;
      M.idx[slot][lane] = ok ? nz.c : -1;
      M.val[slot][lane] = ok ? nz.value(a) : 0.f;
      bad_col |= sl < U && y + mine < e && !ok;
      const int next = y + NG * U + mine;
      nz.load(a, sl < U && next < e, next);
      const bool whole = !LEAN && __all_sync(kFullMask, ok || sl >= U);
      __syncwarp();
      BVec<L> bv[U][K];
      if (whole) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
          const int c = M.idx[slot][grp * G + j];
#pragma unroll
          for (int k = 0; k < K; ++k)
            bv[j][k].load(my_B[k] + (unsigned long long)(unsigned)c * a.ldb);
        }
      } else {
#pragma unroll
        for (int j = 0; j < U; ++j) {
          const int c = M.idx[slot][grp * G + j];
#pragma unroll
          for (int k = 0; k < K; ++k) {
            bv[j][k].zero();
            if (c >= 0) bv[j][k].load(my_B[k] + (unsigned long long)(unsigned)c * a.ldb);
          }
        }
      }
      const int groups = LEAN ? NG : min(NG, (e - y + U - 1) / U);  // with a nonzero of this step
#pragma unroll 1
      for (int g = 0; g < groups; ++g) {
        if (grp == g) {  // a nonzero past the end adds 0 * 0 to a sum that is never -0
#pragma unroll
          for (int j = 0; j < U; ++j) add(M.val[slot][grp * G + j], bv[j], acc);
        }
        __syncwarp();
        if (NG > 1) {
#pragma unroll
          for (int k = 0; k < P; ++k) acc[k] = __shfl_sync(kFullMask, acc[k], g * G + sl);
        }
      }
    }
    if (grp == 0)
      store(a.C + (long long)row * a.ldc + L::column(sl, 0), acc,
            a.row_scale ? __ldg(a.row_scale + row) : 1.f);
    __syncwarp();
  }

  // One block: rows [rs, re), at most kMaxRows, and nonzeros [ns, ne), the rows'
  // ends among them (not ORDERED: at most kMaxNz).  `inside`: row rs began before
  // nonzero ns.  z_out: row rs ends here without a nonzero.  ORDERED: stops
  // before the first row that is long, whose offsets fall or that ends before ns
  // or kMaxNz past it, so that the rows before it end in order; returns the row
  // it stopped at.
  // Leaves every piece's open row in M.open, with M.first, closed, has_pend.
  __device__ __forceinline__ int block(const int rs, int re, const int ns, int ne,
                                       const bool inside, bool& z_out) {
    const float* const scale = a.row_scale;
    int len = ne - ns, nrows = re - rs;
    // pieces: equal shares of the nonzeros in whole steps (ORDERED: moved to
    // row starts below)
    auto share = [&]() { return (len + NG * U - 1) / (NG * U) * U; };
    int per = share();
    const long long y0 = ns + (long long)per * grp;
    int y = y0 < ne ? (int)y0 : ne;
    int ye = y0 + per < ne ? (int)(y0 + per) : ne;
    Nz nz;
    if (!ORDERED) nz.load(a, sl < U && y + sl < ye, y + sl);

    // the row ends as bits; empty rows are written here
    bool dense = true;
    z_out = false;
    for (int i = lane; i < (min(len, kMaxNz) >> 5) + 2; i += 32) M.ends[i] = 0u;
    for (int i = lane; i < (nrows >> 5) + 2; i += 32) M.rowm[i] = 0u;
    __syncwarp();
    for (int i0 = 0; i0 < nrows; i0 += 128) {
      int s4[4], e4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + 32 * u + lane;
        s4[u] = i < nrows ? __ldg(a.offsets + rs + i) : 0;
        e4[u] = i < nrows ? __ldg(a.offsets + rs + i + 1) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i0 + 32 * u >= nrows) break;
        const int i = i0 + 32 * u + lane, s = s4[u], e = e4[u];
        if constexpr (ORDERED) {
          const unsigned most = NG > 1 ? (unsigned)a.long_row : kMaxNz - kBlock;
          const unsigned lm = __ballot_sync(
              kFullMask, i < nrows && ((unsigned)e - (unsigned)s > most ||  // or e < s
                                       (unsigned)e - (unsigned)ns > (unsigned)kMaxNz));
          if (lm) {  // the block ends before this row
            bad_off |= i < nrows && (s < ns || e < s || e > ne);
            const int q = __ffs(lm) - 1;
            nrows = i0 + 32 * u + q;
            ne = min(max(__shfl_sync(kFullMask, s, q), ns), ne);
          }
        }
        const bool empty = i < nrows && s == e;
        const bool z = !ORDERED && i == 0 && inside && e == ns;
        const bool bit = i < nrows && !empty && !z && e > ns && e <= ne && e - ns <= kMaxNz;
        if (bit) {
          const unsigned m = 1u << ((e - ns - 1) & 31);
          bad_off |= (atomicOr(&M.ends[(e - ns - 1) >> 5], m) & m) != 0;
        }
        bad_off |= i < nrows && !empty && !z && (!bit || e < s);
        z_out |= __any_sync(kFullMask, z);
        const unsigned rb = __ballot_sync(kFullMask, bit);
        if (lane == 0) M.rowm[i >> 5] = rb;
        dense = dense && rb == __ballot_sync(kFullMask, i < nrows);
        for (unsigned em = __ballot_sync(kFullMask, empty); em; em &= em - 1) {
          const long long row = rs + i0 + 32 * u + __ffs(em) - 1;
          const float zero = scale ? 0.f * __ldg(scale + row) : 0.f;
          for (int c = lane; c < a.n; c += 32) __stcs(a.C + row * a.ldc + c, zero);
        }
      }
    }
    __syncwarp();
    if (ORDERED) {
      re = rs + nrows;
      if (nrows == 0) return re;
      ne = min(ne, ns + kMaxNz);  // (past the last row's end on malformed offsets alone)
      len = ne - ns;
      per = share();
    }

    // the row each piece starts in
    int x = rs;
    bool began = grp == 0 && inside;
    int before = 0;  // the row ends before this group's piece
#pragma unroll
    for (int p = 1; p < NG; ++p) {
      const int q = min(per * p, len);
      int c = 0;
      for (int i = lane; i <= q >> 5; i += 32) {
        unsigned m = M.ends[i];
        if (i == q >> 5) m &= (1u << (q & 31)) - 1u;
        c += __popc(m);
      }
      c = __reduce_add_sync(kFullMask, c);
      if (p == grp) before = c;
    }
    if (dense) {
      x = rs + before;
    } else {
      // the `before`-th set bit of rowm (re when there is none)
      int skip = before, at = nrows;
      for (int i = 0; i <= nrows >> 5; ++i) {
        const unsigned m = M.rowm[i];
        const int c = __popc(m);
        if (skip >= 0 && skip < c) {
          unsigned t = m;
          for (int k = 0; k < skip; ++k) t &= t - 1;
          at = 32 * i + __ffs(t) - 1;
          skip = -1;
        } else if (skip >= 0) {
          skip -= c;
        }
      }
      x = rs + min(at, nrows);
    }
    if (ORDERED) {
      // whole rows: from row x's start to the next piece's row's
      y = x < re ? min(max(__ldg(a.offsets + x), ns), ne) : ne;
      ye = __shfl_down_sync(kFullMask, y, G);
      if (grp == NG - 1) ye = ne;
      ye = max(y, ye);
      nz.load(a, sl < U && y + sl < ye, y + sl);
    } else if (y > ns) {
      const int q = y - ns - 1;
      began = !((M.ends[q >> 5] >> (q & 31)) & 1u);
    } else {
      began = inside && !z_out;
    }
    const int x0 = x;
    int steps = (ye - y + U - 1) / U;
#pragma unroll
    for (int d = G; d < 32; d <<= 1) steps = max(steps, __shfl_xor_sync(kFullMask, steps, d));

    auto step_ends = [&](int at) -> unsigned {  // the piece's row ends in [at, at + U)
      if (at >= ye) return 0u;
      const int q = at - ns;
      if (!ORDERED) {
        const unsigned b = reinterpret_cast<const unsigned char*>(M.ends)[q >> 3];
        return U == 8 ? b : (b >> (q & 4)) & 15u;
      }
      const int left = ye - at;
      return bits_at(M.ends, q) & ((1u << (left < U ? left : U)) - 1u);
    };
    auto next_row = [&](int r) {  // the next row after r that is not empty
      int nx = r + 1 - rs;
      if (!dense) {
        while (nx < nrows) {
          const unsigned m = M.rowm[nx >> 5] >> (nx & 31);
          if (m) {
            nx += __ffs(m) - 1;
            break;
          }
          nx = (nx & ~31) + 32;
        }
        nx = min(nx, nrows);
      }
      return rs + nx;
    };
    float acc[P];
#pragma unroll
    for (int k = 0; k < P; ++k) acc[k] = 0.f;
    bool has_pend = false;
    // a row's sum is put aside before every kFold-th step unless its group has a
    // row end in that step: short chains of additions, for the rounding error
    // (at most (kFold + 1) U - 1 nonzeros).  Each group for itself: the others'
    // rows may end in every step.
    bool folded = false;
    auto unfold = [&]() {
      if constexpr (!ORDERED) {
        if (folded) {
#pragma unroll
          for (int k = 0; k < P; ++k) acc[k] = __fadd_rn(M.fold[k][lane], acc[k]);
          folded = false;
        }
      }
    };
    float* crow = a.C + (long long)x * a.ldc + L::column(sl, 0);
    float scn = scale ? __ldg(scale + min(x + sl, (int)a.rows - 1)) : 1.f;
    unsigned ends = step_ends(y);
    auto step = [&](int i) {
      const int slot = i & 1;
      const bool ok = (unsigned)nz.c < (unsigned long long)a.cols;
      const bool in = y + sl < ye;
      M.idx[slot][lane] = ok ? nz.c : -1;
      M.val[slot][lane] = ok ? nz.value(a) : 0.f;
      if (scale) M.sc[slot][lane] = scn;
      const bool whole = __all_sync(kFullMask, ok || sl >= U) && a.ldb >> 32 == 0;
      bad_col |= sl < U && in && !ok;
      // the next step's loads go first: the B reads of this one are then the
      // only thing that it waits for
      nz.load(a, sl < U && y + U + sl < ye, y + U + sl);
      int xn = x;
      if (dense)
        xn += __popc(ends);
      else if (ends)
        for (unsigned t = ends; t; t &= t - 1) xn = next_row(xn);
      if (scale) scn = __ldg(scale + min(xn + sl, (int)a.rows - 1));
      __syncwarp();
      BVec<L> b[U][K];
      if (whole) {
        int c[U];
#pragma unroll
        for (int j = 0; j < U; j += 4) {
          const int4 t = *reinterpret_cast<const int4*>(&M.idx[slot][grp * G + j]);
          c[j] = t.x; c[j + 1] = t.y; c[j + 2] = t.z; c[j + 3] = t.w;
        }
#pragma unroll
        for (int j = 0; j < U; ++j)
#pragma unroll
          for (int k = 0; k < K; ++k)
            b[j][k].load(my_B[k] + (unsigned long long)(unsigned)c[j] * (unsigned)a.ldb);
      } else {
#pragma unroll
        for (int j = 0; j < U; ++j) {
          const int c = M.idx[slot][grp * G + j];
#pragma unroll
          for (int k = 0; k < K; ++k) {
            b[j][k].zero();
            if (c >= 0) b[j][k].load(my_B[k] + (unsigned long long)(unsigned)c * a.ldb);
          }
        }
      }
      float v[U];
#pragma unroll
      for (int j = 0; j < U; j += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&M.val[slot][grp * G + j]);
        v[j] = t.x; v[j + 1] = t.y; v[j + 2] = t.z; v[j + 3] = t.w;
      }
      const float* const sc = &M.sc[slot][grp * G];
      if (!__any_sync(kFullMask, ends != 0)) {
#pragma unroll
        for (int j = 0; j < U; ++j) add(v[j], b[j], acc);
      } else {
        // the first row of a piece may be another's too, and a window of rows or
        // scales may not reach the last end: those go one by one
        bool each = ends != 0 && began;
        unsigned rw = 0u;
        if (!dense) {
          rw = bits_at(M.rowm, min(x - rs, nrows));
          const int ne_ = __popc(ends);
          each |= ends != 0 && (!(rw & 1u) || __popc(rw) <= ne_ ||
                                (scale && __popc(rw & (kFullMask >> (32 - G))) < ne_));
        }
        bool any_each = __any_sync(kFullMask, each || (folded && ends != 0));
        if (any_each) {  // a sum put aside is taken up before the step of its row's end
          if (ends) unfold();
          any_each = __any_sync(kFullMask, each);
        }
        if (!any_each) {
          if (dense) {
            if (scale)
              sums<false, true>(b, v, ends, 0u, sc, acc, crow);
            else
              sums<false, false>(b, v, ends, 0u, sc, acc, crow);
          } else {
            if (scale)
              sums<true, true>(b, v, ends, rw, sc, acc, crow);
            else
              sums<true, false>(b, v, ends, rw, sc, acc, crow);
          }
        } else {
          int r = x;
#pragma unroll 1
          for (int j = 0; j < U; ++j) {
            const int c = M.idx[slot][grp * G + j];
            BVec<L> bj[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
              bj[k].zero();
              if (c >= 0) bj[k].load(my_B[k] + (unsigned long long)(unsigned)c * a.ldb);
            }
            add(M.val[slot][grp * G + j], bj, acc);
            if ((ends >> j) & 1u) {
              if (began) {
                if constexpr (!ORDERED) {
#pragma unroll
                  for (int k = 0; k < K; ++k)
#pragma unroll
                    for (int t = 0; t < V; ++t)
                      M.pend[grp][L::column(sl, k) + t] = acc[V * k + t];
                }
                has_pend = true;
                began = false;
              } else {
                store(crow, acc, scale ? __ldg(scale + r) : 1.f);
              }
#pragma unroll
              for (int k = 0; k < P; ++k) acc[k] = 0.f;
              const int nr = next_row(r);
              crow += (nr - r) * a.ldc;
              r = nr;
            }
          }
        }
      }
      x = xn;
      y = min(y + U, ye);
      ends = step_ends(y);
    };
#pragma unroll 1
    for (int i0 = 0; i0 < steps; i0 += kFold) {
      if constexpr (!ORDERED) {
        if (i0 > 0 && ends == 0) {
#pragma unroll
          for (int k = 0; k < P; ++k) {
            M.fold[k][lane] = folded ? __fadd_rn(M.fold[k][lane], acc[k]) : acc[k];
            acc[k] = 0.f;
          }
          folded = true;
        }
      }
      const int i1 = min(i0 + kFold, steps);
#pragma unroll 1
      for (int i = i0; i < i1; ++i) step(i);
    }
    unfold();
    __syncwarp();
    if constexpr (!ORDERED) {
      if (sl == 0) {
        M.first[grp] = x0;
        M.closed[grp] = x > x0;
        M.has_pend[grp] = has_pend;
      }
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int t = 0; t < V; ++t) M.open[grp][L::column(sl, k) + t] = acc[V * k + t];
      __syncwarp();
    }
    return re;
  }
};

template <typename L, bool ORDERED>
__global__ void __launch_bounds__(kTPB, kMinCtas) spmm_kernel(const Args a) {
  using Sm = Smem<L, ORDERED>;
  constexpr int NG = 32 / L::G;
  constexpr int Q = (L::kCols + 31) / 32;  // columns per lane when rows are stitched
  __shared__ Sm smem[kWarps];
  __shared__ unsigned s_ticket[2];
  Sm& M = smem[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  long long w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  unsigned tag = 0;
  if (!ORDERED) {
    // one ticket per CTA: a range only waits on ranges of CTAs that are
    // running
    if (threadIdx.x == 0) take_ticket(a.hdr, gridDim.x, &s_ticket[0], &s_ticket[1]);
    __syncthreads();
    w = (long long)s_ticket[0] * kWarps + (threadIdx.x >> 5);
    tag = epoch_tag(s_ticket[1]);
  }
  if (w >= a.num_ranges) return;
  const long long total = (long long)kRowItems * a.rows + a.nnz;
  const long long d0 = min(w * a.range_items, total), d1 = min(d0 + a.range_items, total);
  Walk<L, ORDERED> walk(a, M);
  float run[Q], pend[Q];  // the open row's partial; row r0's part of this range
  bool any_closed = false, wait_row = false;  // wait_row: row r0 is ours to finish
#pragma unroll
  for (int q = 0; q < Q; ++q) run[q] = pend[q] = 0.f;
  int r0 = 0, n0 = 0, off_r0 = 0, re = 0, ne = 0, off_re = 0;
  for (long long d = d0; d < d1; d += a.block_items) {
    SplitPoint sa, sb;
    const long long db = min(d + a.block_items, d1);
    warp_merge_search2_w([&](long long k) { return __ldg(a.offsets + 1 + k); }, a.rows, a.nnz, d,
                         db, kRowItems, sa, sb);
    int rs = (int)sa.x, ns = split_nonzero(sa, d, kRowItems, a.rows);
    re = (int)sb.x;
    ne = split_nonzero(sb, db, kRowItems, a.rows);
    off_re = sb.start;
    // on malformed offsets the two split points are unrelated
    const int re_in = min(max(re, rs), rs + kMaxRows);
    if (re != re_in) raise_flag(a.hdr, EL_FLAG_OFFSETS, (unsigned)rs);
    re = re_in;
    bool z = false;
    if (ORDERED) {  // whole rows
      const int m = (int)a.nnz;
      ns = min(max(sa.start, 0), m);
      ne = min(max(sb.start, ns), m);
      while (rs < re) {  // runs of shorter rows, and each long row by itself
        rs = walk.block(rs, re, ns, ne, false, z);
        if (rs >= re) break;
        const int b = min(max(__ldg(a.offsets + rs), ns), ne);
        ns = min(max(__ldg(a.offsets + rs + 1), b), ne);
        walk.template whole_row<true>(rs++, b, ns);
      }
    } else {
      if (d == d0) {
        r0 = rs;
        n0 = ns;
        off_r0 = sa.start;
      }
      const int ne_in = min(max(ne, ns), ns + kMaxNz);
      if (ne != ne_in) raise_flag(a.hdr, EL_FLAG_OFFSETS, (unsigned)rs);
      ne = ne_in;
      walk.block(rs, re, ns, ne, ns > sa.start, z);
      // stitch the rows that cross pieces, in piece order
      const bool need_lb = n0 > off_r0;
      if (z) {  // row rs ended at the block's first nonzero
        const float sc = a.row_scale ? __ldg(a.row_scale + rs) : 1.f;
        const bool lb = need_lb && !any_closed;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int c = lane + 32 * q;
          if (lb)
            pend[q] = run[q];
          else if (c < a.n)
            a.C[(long long)rs * a.ldc + c] = run[q] * sc;
          run[q] = 0.f;
        }
        wait_row |= lb;
        any_closed = true;
      }
      for (int s = 0; s < NG; ++s) {
        const bool hp = M.has_pend[s], cl = M.closed[s], lb = hp && need_lb && !any_closed;
        const long long row = M.first[s];
        const float sc = hp && a.row_scale ? __ldg(a.row_scale + row) : 1.f;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int c = lane + 32 * q;
          if (c >= a.n) continue;
          if (hp) {
            const float t = __fadd_rn(run[q], M.pend[s][c]);
            if (lb)
              pend[q] = t;
            else
              a.C[row * a.ldc + c] = t * sc;
          }
          run[q] = cl ? M.open[s][c] : __fadd_rn(run[q], M.open[s][c]);
        }
        wait_row |= lb;
        any_closed |= cl;
      }
      __syncwarp();
    }
  }
  if (walk.bad_off) raise_flag(a.hdr, EL_FLAG_OFFSETS, (unsigned)re);
  if (walk.bad_col) raise_flag(a.hdr, EL_FLAG_INDEX_RANGE, (unsigned)re);
  if constexpr (!ORDERED) {
    // publish the open row's partial vector if this range holds any of it
    if (re < a.rows && ne > max(off_re, n0)) {
      float* const dst = a.vec + w * kPassCols;
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (lane + 32 * q < a.n) __stcg(dst + lane + 32 * q, run[q]);
      __threadfence();
      __syncwarp();
      if (lane == 0 && !(a.test_hooks & 1)) st_release_u32(&a.flags[w].flag, tag);
    }
    if (wait_row) {
      // row r0 began in range `first`: add the partials of ranges [first, w)
      // in order, 32 flags polled at a time
      const long long first = max(0LL, ((long long)kRowItems * r0 + off_r0) / a.range_items);
      float chain[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) chain[q] = 0.f;
      bool ok = true;
      for (long long base = first; base < w && ok; base += 32) {
        if (base + lane < w) {
          const unsigned* const f = &a.flags[base + lane].flag;
          if (ld_acquire_u32(f) != tag) {
            const uint64_t t0 = global_timer_ns();
            while (ld_acquire_u32(f) != tag) {
              if (global_timer_ns() - t0 > a.wait_ns) {
                ok = false;
                break;
              }
              __nanosleep(100);
            }
          }
        }
        ok = __all_sync(kFullMask, ok);
        if (!ok) break;
        // the lanes' acquires come before every lane's reads of the vectors
        // (a vote alone orders no memory)
        __syncwarp();
        const int cnt = (int)(w - base < 32 ? w - base : 32);
#pragma unroll 8
        for (int k = 0; k < cnt; ++k) {
          const float* const src = a.vec + (base + k) * kPassCols;
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (lane + 32 * q < a.n) chain[q] = __fadd_rn(chain[q], __ldcg(src + lane + 32 * q));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) raise_flag(a.hdr, EL_FLAG_TIMEOUT, 6);
      const float sc = a.row_scale ? __ldg(a.row_scale + r0) : 1.f;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int c = lane + 32 * q;
        if (c < a.n) a.C[(long long)r0 * a.ldc + c] = __fadd_rn(chain[q], pend[q]) * sc;
      }
    }
  }
}

// --------------------------------------------------------------- few rows
// ORDERED, a matrix of few rows: a warp per row, 32 / G x U of its B rows in
// flight at once.  A row of 30 nonzeros is then one or two round trips; the
// walk's range of a few rows is its split search, its row ends and a chain of
// U nonzeros per step in one group of the warp, the other groups idle.  Up to
// kFewRows rows per resident warp of the walk (3 where a lane holds 8 columns,
// whose hand-over from group to group costs twice as much).  FP32 B, n = 8, the
// walk / a warp per row: 5,276 rows of 38 11 / 7 us, 15,802 13-22 / 14, 52,644
// 22 / 42; 13,346 of 15 10 / 7, 40,013 14 / 17; 15,013 of 4 7 / 6, 50,013
// 9 / 15; 27-point stencil 8,000 rows 12 / 6, 21,952 15 / 15; log-normal rows of
// 12, 16,679 27 / 22, 50,013 32 / 33.  BF16 B, n = 16 (8 columns per lane):
// 8,000 stencil rows 14 / 9, 13,346 of 15 11 / 10, 15,802 of 38 17 / 21.
constexpr int kFewRows = 5, kFewRowsWide = 3;
template <typename L>
__global__ void __launch_bounds__(kTPB, kMinCtas) warp_rows_kernel(const Args a) {
  __shared__ RowSmem smem[kWarps];
  Walk<L, true, RowSmem> walk(a, smem[threadIdx.x >> 5]);
  const int nnz = (int)a.nnz;
  const long long step = (long long)gridDim.x * kWarps;
  auto bound = [&](long long r) { return __ldg(a.offsets + min(r, a.rows)); };
  long long row = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  int b = bound(row), e = bound(row + 1);
  for (; row < a.rows; row += step) {  // warp-uniform
    // the next row's bounds are in flight meanwhile
    const int nb = bound(row + step), ne = bound(row + step + 1);
    walk.bad_off |= b < 0 || e < b || e > nnz;
    const int lo = min(max(b, 0), nnz);
    walk.template whole_row<false>((int)row, lo, min(max(e, lo), nnz));
    b = nb;
    e = ne;
  }
  if (walk.bad_off) raise_flag(a.hdr, EL_FLAG_OFFSETS, 0);
  if (walk.bad_col) raise_flag(a.hdr, EL_FLAG_INDEX_RANGE, 0);
}

template <typename L>
bool few_rows(const SpmmCall& c) {
  const long long warps = (long long)device_info(c.device).sm_count * kMinCtas * kWarps;
  return c.A.rows <= warps * (L::P <= 4 ? kFewRows : kFewRowsWide);
}

template <typename L>
el_status launch_warp_rows(const SpmmCall& c, const Args& a) {
  const int per_sm = resident_ctas_per_sm((const void*)warp_rows_kernel<L>, kTPB, 0);
  const long long most = (long long)(per_sm > 0 ? per_sm : 1) * device_info(c.device).sm_count;
  const long long need = (a.rows + kWarps - 1) / kWarps;
  warp_rows_kernel<L><<<(unsigned)(need < most ? need : most), kTPB, 0, c.stream>>>(a);
  return cuda_status(cudaGetLastError(), "spmm launch");
}

// ------------------------------------------------------------- narrow B, C
// thread_mapped with NC <= kNarrow columns: a thread per row, the row walked
// once, W nonzeros' values and B elements in flight with the next W's
// columns.  A B row is then less than the sectors it lies in, neighbouring
// rows of a banded matrix share them in L1, and the row ends of the walk above
// cost as much as for wide rows.  2M nonzeros, FP32, walk / thread per row:
// 27-point stencil n = 1 29 / 10 us, n = 4 28 / 14; n = 4 in log-normal rows of
// 4 59 / 32, uniform rows of 38 28 / 30, log-normal rows of 38 77 / 98.  The line
// is by n alone: where rows are long the thread per row loses up to a quarter,
// where they are short the walk loses half, and how the lengths vary, which
// decides between them from 6 columns on (n = 6: stencil 27 / 12, uniform rows of
// 38 25 / 34, log-normal rows of 27 76 / 106, of 4 65 / 43), is not known here.  So
// from 6 columns on the walk keeps rows of every length balanced, and a stencil
// of more rows than the warp per row takes is slower than by a thread per row
// (22,000 rows, n = 6: 16 / 6).
constexpr int kNarrow = 5;
template <typename VT, typename BT, int NC>
__global__ void __launch_bounds__(256, 3) thread_rows_kernel(const Args a) {
  constexpr int W = NC == 1 ? 16 : 8;
  const VT* const vals = reinterpret_cast<const VT*>(a.values);
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < a.rows;
       row += (long long)gridDim.x * blockDim.x) {
    int b = __ldg(a.offsets + row), e = __ldg(a.offsets + row + 1);
    if (b < 0 || e > a.nnz || e < b) {
      raise_flag(a.hdr, EL_FLAG_OFFSETS, (unsigned)row);
      b = min(max(b, 0), (int)a.nnz);
      e = min(max(e, b), (int)a.nnz);
    }
    const float scale = a.row_scale ? __ldg(a.row_scale + row) : 1.f;
    bool bad = false;
    float sum[NC];
    int c[W];
#pragma unroll
    for (int j = 0; j < NC; ++j) sum[j] = 0.f;
    const int len = e - b;
    const int* const idx = a.indices + b;
    const VT* const val = vals + b;
#pragma unroll
    for (int k = 0; k < W; ++k) c[k] = k < len ? __ldg(idx + k) : -1;
    for (int q = 0; q < len; q += W) {
      float v[W], bv[W][NC];
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const bool ok = (unsigned)c[k] < (unsigned)a.cols;
        bad |= !ok && k < len - q;
        v[k] = ok ? to_f32(val[q + k]) : 0.f;
        const BT* const r =
            reinterpret_cast<const BT*>(a.B + (ok ? (unsigned)c[k] * a.ldb : 0ull));
#pragma unroll
        for (int j = 0; j < NC; ++j) bv[k][j] = ok ? to_f32(r[j]) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < W; ++k) c[k] = k < len - q - W ? __ldg(idx + q + W + k) : -1;
#pragma unroll
      for (int k = 0; k < W; ++k)
        if (k < len - q) {
#pragma unroll
          for (int j = 0; j < NC; ++j) sum[j] = __fadd_rn(sum[j], __fmul_rn(v[k], bv[k][j]));
        }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j)
      a.C[row * a.ldc + j] = a.row_scale ? sum[j] * scale : sum[j];
    if (bad) raise_flag(a.hdr, EL_FLAG_INDEX_RANGE, (unsigned)row);
  }
}

template <typename VT, typename BT>
el_status launch_thread_rows(const SpmmCall& c, const Args& a) {
  const long long most = (long long)device_info(c.device).sm_count * 32;
  const long long need = (a.rows + 255) / 256;
  const unsigned grid = (unsigned)(need < most ? need : most);
  switch (a.n) {
    case 1: thread_rows_kernel<VT, BT, 1><<<grid, 256, 0, c.stream>>>(a); break;
    case 2: thread_rows_kernel<VT, BT, 2><<<grid, 256, 0, c.stream>>>(a); break;
    case 3: thread_rows_kernel<VT, BT, 3><<<grid, 256, 0, c.stream>>>(a); break;
    case 4: thread_rows_kernel<VT, BT, 4><<<grid, 256, 0, c.stream>>>(a); break;
    default: thread_rows_kernel<VT, BT, kNarrow><<<grid, 256, 0, c.stream>>>(a); break;
  }
  return cuda_status(cudaGetLastError(), "spmm launch");
}

// ----------------------------------------------------------------- launch
template <typename L, bool ORDERED>
el_status launch_kernel(const SpmmCall& c, Args a) {
  auto kern = spmm_kernel<L, ORDERED>;
  const int per_sm = resident_ctas_per_sm((const void*)kern, kTPB, 0);
  long long warps = (long long)(per_sm > 0 ? per_sm : 1) * device_info(c.device).sm_count * kWarps;
  if (!ORDERED) {
    const long long most = (long long)(c.scratch_bytes / (kPassCols * sizeof(float)));
    warps = warps < most ? warps : most;
    warps = warps < c.ws.nslots ? warps : c.ws.nslots;
    if (warps < 1) return fail(EL_ERR_INVALID_ARGUMENT, "spmm merge_path: workspace too small");
  }
  const long long total = (long long)kRowItems * a.rows + a.nnz;
  long long ri = (total + warps - 1) / warps;
  if (ri < 64) ri = 64;
  a.range_items = ri;
  const long long blocks = (ri + kBlock - 1) / kBlock;
  a.block_items = (int)((ri + blocks - 1) / blocks);
  a.long_row = ri >= kLongRow ? kLongRow : ri > 128 ? (int)ri / 4 : 32;
  a.num_ranges = (total + ri - 1) / ri;
  const long long grid = (a.num_ranges + kWarps - 1) / kWarps;
  kern<<<(unsigned)grid, kTPB, 0, c.stream>>>(a);
  return cuda_status(cudaGetLastError(), "spmm launch");
}

template <typename BT, int V, int K, int G>
el_status launch_pass(const SpmmCall& c, const Args& a, bool ordered) {
  using L = Lay<BT, V, K, G>;
  if (ordered && few_rows<L>(c)) return launch_warp_rows<L>(c, a);
  return ordered ? launch_kernel<L, true>(c, a) : launch_kernel<L, false>(c, a);
}

template <typename BT>
el_status launch(const SpmmCall& c, int schedule) {
  constexpr int kB = (int)sizeof(BT);
  const bool ordered = schedule != EL_SCHED_MERGE_PATH_FLAT;
  Args a;
  a.rows = c.A.rows;
  a.cols = c.A.cols;
  a.nnz = c.A.nnz;
  a.offsets = c.A.offsets;
  a.indices = c.A.indices;
  a.values = reinterpret_cast<const unsigned char*>(c.A.values);
  a.value_dtype = c.A.value_dtype;
  a.row_scale = c.A.row_scale;
  a.B = reinterpret_cast<const unsigned char*>(c.B);
  a.ldb = (unsigned long long)c.ldb * kB;
  a.ldc = c.ldc;
  a.hdr = c.ws.hdr;
  a.flags = c.ws.slots;
  a.vec = reinterpret_cast<float*>(c.scratch);
  a.wait_ns = c.wait_ns;
  a.test_hooks = c.o.test_hooks;
  if (schedule == EL_SCHED_THREAD_MAPPED && c.n <= kNarrow) {
    a.n = (int)c.n;
    a.b_first = 0;
    a.C = c.C;
    if (a.value_dtype == EL_F32) return launch_thread_rows<float, BT>(c, a);
    if constexpr (kB == 4) {
      return a.value_dtype == EL_BF16 ? launch_thread_rows<__nv_bfloat16, BT>(c, a)
                                      : launch_thread_rows<__half, BT>(c, a);
    } else {  // 16-bit values come with B of their own type alone
      return launch_thread_rows<BT, BT>(c, a);
    }
  }
  // columns per load: the widest vectors on whose boundaries every row of B
  // and C starts and of which n is a multiple
  int v = 16 / kB;
  for (; v > 1; v /= 2) {
    const int f = v < 4 ? v : 4;  // floats per store
    if (c.n % v == 0 && c.ldb % v == 0 && (uintptr_t)c.B % (v * kB) == 0 && c.ldc % f == 0 &&
        (uintptr_t)c.C % (4 * f) == 0)
      break;
  }
  for (long long cb = 0; cb < c.n; cb += kPassCols) {
    a.n = (int)(c.n - cb < kPassCols ? c.n - cb : kPassCols);
    a.b_first = (unsigned long long)cb * kB;
    a.C = c.C + cb;
    const int n = a.n;
    el_status s = EL_OK;
    if (v == 8) {
      if constexpr (kB == 2)
        s = n <= 32   ? launch_pass<BT, 8, 1, 4>(c, a, ordered)
            : n <= 64 ? launch_pass<BT, 8, 1, 8>(c, a, ordered)
                      : launch_pass<BT, 8, 1, 16>(c, a, ordered);
    } else if (v == 4) {
      s = n <= 16   ? launch_pass<BT, 4, 1, 4>(c, a, ordered)
          : n <= 32 ? launch_pass<BT, 4, 1, 8>(c, a, ordered)
          : n <= 64 ? launch_pass<BT, 4, 1, 16>(c, a, ordered)
                    : launch_pass<BT, 4, 1, 32>(c, a, ordered);
    } else if (v == 2) {
      s = n <= 16   ? launch_pass<BT, 2, 2, 4>(c, a, ordered)
          : n <= 32 ? launch_pass<BT, 2, 2, 8>(c, a, ordered)
          : n <= 64 ? launch_pass<BT, 2, 2, 16>(c, a, ordered)
                    : launch_pass<BT, 2, 2, 32>(c, a, ordered);
    } else {
      s = n <= 8    ? launch_pass<BT, 1, 2, 4>(c, a, ordered)
          : n <= 16 ? launch_pass<BT, 1, 2, 8>(c, a, ordered)
          : n <= 32 ? launch_pass<BT, 1, 2, 16>(c, a, ordered)
          : n <= 64 ? launch_pass<BT, 1, 2, 32>(c, a, ordered)
          : n <= 96 ? launch_pass<BT, 1, 3, 32>(c, a, ordered)
                    : launch_pass<BT, 1, 4, 32>(c, a, ordered);
    }
    if (s != EL_OK) return s;
  }
  return EL_OK;
}

}  // namespace spmm

template <typename BT>
el_status spmm_launch(const SpmmCall& c, int schedule) {
  return spmm::launch<BT>(c, schedule);
}

#define EL_INSTANTIATE_SPMM(BT) template el_status spmm_launch<BT>(const SpmmCall&, int);

}  // namespace el
