// csr_build.cu -- el_csr_from_coo: COO (device) -> CSR (device), the
// reference's CSR construction [include/loops/container/csr.hxx:86-94]:
// sort the entries by (row, column) [coo.hxx:104-113, :145-148], take the
// column indices and values in that order, and offsets[r] = the first
// sorted position whose row is >= r [detail/convert.hxx:75-77].
//
// Entries with equal (row, column) keep their input order -- the reference's
// thrust sort leaves their order unspecified and keeps them all, and so does
// this.  Entries whose row or column is outside the matrix are an error
// (EL_ERR_MALFORMED_CSR), found before anything is written.
//
// Two ways to the same arrays:
//
//  window sort: the row lengths are counted and summed, which gives the
//    offsets, i.e. where each row's entries go.  One pass moves every entry to
//    the window of W consecutive places that its row starts in (an entry of a
//    row longer than a window's spare room: that its column c suggests, s +
//    floor(c L / cols) for a row of L entries from s on), and one CTA per
//    window sorts it in shared memory: a counting sort by the place that the
//    entry's column suggests between its row's first and last one, then a
//    rank among the few entries that share a place.  A window has room for
//    1.5 to 2 W entries; a matrix that overfills one (a long row whose columns
//    crowd together) goes the other way.
//  radix sort (cub::DeviceRadixSort) of the key row << bits | column.
//
// Measured, whole call: 15.4M shuffled entries of a 2^20-row power-law matrix
// 1128 us by the radix sort of a 51-bit key (7 passes of 120 us, values
// gathered 102 us, offsets searched 33 us), 627 us by the window sort (count
// 87, sums 12, move 242, sort 278 us).  Uniform entries in rows of 15: 200,000
// 147 -> 70 us, 2M 275 -> 147, 8M 669 -> 333, 15M 1124 -> 638.  A twentieth of the
// entries in one row's few columns, which overfills a window and goes to the
// radix sort of a 40-bit key: 200,000 147 -> 143, 2M 273 -> 274, 8M 668 -> 620, 15M
// 1120 -> 1027.
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

#include "el_internal.h"

namespace el {
namespace {

// --------------------------------------------------------------- radix sort
// key = row << cbits | column
__global__ void keys_kernel(const int32_t* __restrict__ ri, const int32_t* __restrict__ ci,
                            long long nnz, long long rows, long long cols, int cbits,
                            unsigned long long* __restrict__ keys, int32_t* __restrict__ pos,
                            unsigned* __restrict__ bad) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (long long)gridDim.x * blockDim.x) {
    const int r = ri[k], c = ci[k];
    if ((unsigned long long)(unsigned)r >= (unsigned long long)rows ||
        (unsigned long long)(unsigned)c >= (unsigned long long)cols)
      atomicOr(bad, 1u);
    keys[k] = ((unsigned long long)(unsigned)r << cbits) | (unsigned)c;
    pos[k] = (int32_t)k;
  }
}

__global__ void gather_kernel(const unsigned long long* __restrict__ keys,
                              const int32_t* __restrict__ pos, const float* __restrict__ vin,
                              long long nnz, int cbits, int32_t* __restrict__ indices,
                              float* __restrict__ values) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (long long)gridDim.x * blockDim.x) {
    indices[k] = (int32_t)(keys[k] & ((1ull << cbits) - 1ull));
    values[k] = vin[pos[k]];
  }
}

// offsets[r] = number of sorted entries with row < r
__global__ void offsets_kernel(const unsigned long long* __restrict__ keys, long long nnz,
                               long long rows, int cbits, int32_t* __restrict__ offsets) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r <= rows;
       r += (long long)gridDim.x * blockDim.x) {
    const unsigned long long key = (unsigned long long)r << cbits;
    long long lo = 0, hi = nnz;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (keys[mid] < key) lo = mid + 1; else hi = mid;
    }
    offsets[r] = (int32_t)lo;
  }
}

int bits_for(long long n) {  // bits to hold values 0 .. n-1
  int b = 1;
  while (b < 62 && (1LL << b) < n) ++b;
  return b;
}

size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }

// -------------------------------------------------------------- window sort
// Row lengths by atomics, and the range check.  Atomics on one address run
// one after the other (about 1.8 ns each), so a long row would set the time
// (100,000 entries: 180 us).  Each CTA counts the rows that come to it first
// in a table in shared memory, a slot per row, and the rest in global memory:
// a row that comes often soon has a slot.  15.4M power-law entries of 2^20 rows
// 87 us, of which the global atomics take 77 (eight counters per row without a
// table: 137, and 26 more in the sums).  SMALL: few rows, all counted in shared
// memory.
constexpr int kSmallRows = 8192;
constexpr int kCountThreads = 1024;
constexpr int kTableLog = 12;
template <bool SMALL>
__global__ void __launch_bounds__(kCountThreads, 2)
    count_rows_kernel(const int32_t* __restrict__ ri, const int32_t* __restrict__ ci, int nnz,
                      unsigned rows, unsigned cols, unsigned* __restrict__ len,
                      unsigned* __restrict__ flags) {
  constexpr int kSlots = SMALL ? kSmallRows : 1 << kTableLog;
  constexpr unsigned kEmpty = 0xffffffffu;
  __shared__ unsigned s_len[kSlots], s_row[SMALL ? 1 : kSlots];
  for (int i = threadIdx.x; i < (SMALL ? (int)rows : kSlots); i += kCountThreads) {
    s_len[i] = 0u;
    if (!SMALL) s_row[i] = kEmpty;
  }
  __syncthreads();
  auto add = [&](unsigned r, unsigned v) {
    if (SMALL) {
      atomicAdd(s_len + r, v);
      return;
    }
    const unsigned h = r * 0x9e3779b1u >> (32 - kTableLog);
    unsigned own = *const_cast<volatile unsigned*>(s_row + h);
    if (own == kEmpty) {
      own = atomicCAS(s_row + h, kEmpty, r);
      if (own == kEmpty) own = r;
    }
    if (own == r)
      atomicAdd(s_len + h, v);
    else
      atomicAdd(len + r, v);
  };
  const int step = gridDim.x * kCountThreads;  // 4 steps past nnz (at most 2^27) fit an int
  // warp-uniform: k0 - lane counts
  for (int k0 = blockIdx.x * kCountThreads + threadIdx.x; k0 - (int)(threadIdx.x & 31) < nnz;
       k0 += 4 * step) {
    int r[4], c[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + u * step;
      r[u] = k < nnz ? __ldcs(ri + k) : -1;
      c[u] = k < nnz ? __ldcs(ci + k) : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool ok = (unsigned)r[u] < rows && (unsigned)c[u] < cols;
      if (!ok && k0 + u * step < nnz) atomicOr(flags, 1u);
      // entries in row order: one atomic for a warp in one row
      const int r0 = __shfl_sync(kFullMask, r[u], 0);
      const bool same = ok && r[u] == r0;
      if (__all_sync(kFullMask, same)) {
        if ((threadIdx.x & 31) == 0) add(r0, 32u);
      } else if (ok) {
        add(r[u], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (SMALL ? (int)rows : kSlots); i += kCountThreads)
    if (s_len[i]) atomicAdd(len + (SMALL ? (unsigned)i : s_row[i]), s_len[i]);
}

// Row starts: exclusive sums of the lengths of rows 0 .. rows (a last one of
// 0), in blocks of kScan: the blocks' totals, their exclusive sums (one CTA),
// then each block's own, written as (start, length).
constexpr int kScanThreads = 256, kScanPer = 16, kScan = kScanThreads * kScanPer;

// Exclusive sum over the CTA of one value per thread; *total = the sum.
template <int THREADS>
__device__ __forceinline__ unsigned cta_exclusive(unsigned v, unsigned* total) {
  __shared__ unsigned s_sum[THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned t = __shfl_up_sync(kFullMask, inc, d);
    if (lane >= d) inc += t;
  }
  __syncthreads();  // s_sum of an earlier call has been read
  if (lane == 31) s_sum[w] = inc;
  __syncthreads();
  unsigned before = 0, all = 0;
  for (int i = 0; i < THREADS / 32; ++i) {
    const unsigned t = s_sum[i];
    before += i < w ? t : 0u;
    all += t;
  }
  *total = all;
  return before + inc - v;
}

__global__ void __launch_bounds__(kScanThreads)
    block_sums_kernel(const unsigned* __restrict__ len, long long n, unsigned* __restrict__ sums) {
  const long long base = (long long)blockIdx.x * kScan;
  unsigned v = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    const long long k = base + i * kScanThreads + threadIdx.x;
    v += k < n ? __ldg(len + k) : 0u;
  }
  unsigned total;
  cta_exclusive<kScanThreads>(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) scan_sums_kernel(unsigned* sums, int n) {
  unsigned run = 0;
  for (int base = 0; base < n; base += 1024) {
    const int k = base + threadIdx.x;
    unsigned total;
    const unsigned ex = cta_exclusive<1024>(k < n ? sums[k] : 0u, &total);
    if (k < n) sums[k] = run + ex;
    run += total;
  }
}

__global__ void __launch_bounds__(kScanThreads)
    apply_sums_kernel(const unsigned* __restrict__ len, long long n,
                      const unsigned* __restrict__ sums, bool summed, uint2* __restrict__ row) {
  __shared__ unsigned s[kScan + kScan / 32];  // a word of padding per 32: conflict-free both ways
  auto at = [](int i) { return i + (i >> 5); };
  const long long base = (long long)blockIdx.x * kScan;
  const int t = threadIdx.x;
  unsigned mine[kScanPer];  // lengths of the rows this thread writes
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    const long long k = base + i * kScanThreads + t;
    mine[i] = k < n ? __ldg(len + k) : 0u;
    s[at(i * kScanThreads + t)] = mine[i];
  }
  __syncthreads();
  unsigned v[kScanPer], sum = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    v[i] = s[at(t * kScanPer + i)];
    sum += v[i];
  }
  unsigned total, before;  // entries of earlier blocks
  if (summed)
    before = sums[blockIdx.x];
  else  // at most kScanThreads blocks: their totals are summed here
    cta_exclusive<kScanThreads>(t < (int)blockIdx.x ? sums[t] : 0u, &before);
  unsigned run = cta_exclusive<kScanThreads>(sum, &total) + before;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    s[at(t * kScanPer + i)] = run;
    run += v[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    const long long k = base + i * kScanThreads + t;
    if (k < n) row[k] = make_uint2(s[at(i * kScanThreads + t)], mine[i]);
  }
}

constexpr unsigned kHeavy = 0x80000000u;  // an entry of a row that is not kept whole
// Windows of 2^LOGW places with room for kCap entries each.
template <int LOGW>
struct Win {
  static constexpr int W = 1 << LOGW;
  static constexpr int kThreads = LOGW >= 13 ? 1024 : 256;       // of the sort
  static constexpr int kPer = LOGW >= 13 ? 12 : 16;              // its entries per thread
  static constexpr int kCap = kThreads * kPer;
  static constexpr int kLight = kCap - W;       // rows kept whole: entries at most
  static constexpr int kLarge = kCap / 97 + 1;  // places with more than kRankMax entries
  static constexpr int kSmem = kCap * 8 + (kCap + 1) * 4 + kLarge * 8 + 64;
  static_assert(kCap * 8 >= 3 * W * 4, "the rows' counts and column ranges fit the keys' room");
};
constexpr int kMoveThreads = 512, kMovePer = 8, kMoveTile = kMoveThreads * kMovePer;
// A window's fill counter has a 128-byte line of its own: atomics on one line
// run at about 0.3 per ns.
constexpr int kFillStride = 32;
constexpr int kMaxWindows = 16384;  // two counters each in a CTA of the move (128 KB)
constexpr long long kSmallNnz = 1 << 21;
constexpr int kRankMax = 96;    // entries of one place ranked by comparison, at most
constexpr int kWarpSort = 1024;  // of one place sorted by a warp, at most

// The move: every entry goes to its window's region as (row start, or kHeavy |
// place, column, position in the COO, value), in no particular order.  A CTA counts its
// entries per window in shared memory, puts them there in window order,
// reserves room in each window with one atomic and writes them out, so that a
// window's entries leave in one run: one by one, 15.5M 16-byte writes to
// scattered places take 230 us of a 330 us move, in runs of 2-4 the whole move
// 245 us.  flags[1]: a window is full.
template <int LOGW>
__global__ void __launch_bounds__(kMoveThreads, 2)
    move_kernel(const int32_t* __restrict__ ri, const int32_t* __restrict__ ci,
                const float* __restrict__ vin, long long nnz, long long rows, long long cols,
                const uint2* __restrict__ row, int windows, unsigned* __restrict__ fill,
                uint4* __restrict__ recs, unsigned* __restrict__ flags) {
  using Wn = Win<LOGW>;
  constexpr int T = kMoveThreads, P = kMovePer;
  extern __shared__ __align__(16) unsigned char dyn[];
  uint4* const buf = reinterpret_cast<uint4*>(dyn);                          // the tile by window
  unsigned* const count = reinterpret_cast<unsigned*>(dyn + kMoveTile * 16);  // per window
  unsigned* const first = count + windows;  // its first place in buf
  const float inv = 1.f / (float)cols;
  constexpr int kNone = -1;  // no entry (as a heavy place: past every one)
  auto window = [](int e) { return e == kNone ? -1 : (int)(((unsigned)e & ~kHeavy) >> LOGW); };
  for (int i = threadIdx.x; i < windows; i += T) count[i] = 0u;
  const long long base = (long long)blockIdx.x * kMoveTile;
  int est[P], c[P];
  float v[P];
  unsigned at[P];
  const unsigned full = *const_cast<volatile unsigned*>(flags + 1);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const long long k = base + i * T + threadIdx.x;
    est[i] = k < nnz ? __ldcs(ri + k) : -1;
    c[i] = k < nnz ? __ldcs(ci + k) : -1;
    v[i] = k < nnz ? __ldcs(vin + k) : 0.f;
  }
  // a window is full: the radix sort it is, so nothing more is moved
  if (__syncthreads_or(full != 0u)) return;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int r = est[i];
    est[i] = kNone;
    if ((unsigned long long)(unsigned)r < (unsigned long long)rows &&
        (unsigned long long)(unsigned)c[i] < (unsigned long long)cols) {
      const uint2 sl = __ldg(row + r);
      const int s = (int)sl.x, len = (int)sl.y;
      // never decreases with the column: each step rounds monotonically
      const int e = (int)((float)c[i] * ((float)len * inv));
      est[i] = len <= Wn::kLight ? s : (int)(kHeavy | (unsigned)(s + min(e, len - 1)));
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    at[i] = 0;
    const int b = window(est[i]);
    // entries in row order put a whole warp in one window
    const int b0 = __shfl_sync(kFullMask, b, 0);
    if (__all_sync(kFullMask, b == b0)) {
      if (b >= 0) {
        unsigned n = 0;
        if ((threadIdx.x & 31) == 0) n = atomicAdd(&count[b], 32u);
        at[i] = __shfl_sync(kFullMask, n, 0) + (threadIdx.x & 31);
      }
    } else if (b >= 0) {
      at[i] = atomicAdd(&count[b], 1u);
    }
  }
  __syncthreads();
  const int per = (windows + T - 1) / T;  // consecutive windows per thread
  const int w0 = min((int)threadIdx.x * per, windows), w1 = min(w0 + per, windows);
  unsigned sum = 0, total;
  for (int i = w0; i < w1; ++i) sum += count[i];
  unsigned run = cta_exclusive<T>(sum, &total);
  for (int i = w0; i < w1; ++i) {
    first[i] = run;
    run += count[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < P; ++i)
    if (est[i] != kNone)
      buf[first[window(est[i])] + at[i]] =
          make_uint4((unsigned)est[i], (unsigned)c[i],
                     (unsigned)(base + i * T + threadIdx.x), __float_as_uint(v[i]));
  for (int i0 = threadIdx.x; i0 < windows; i0 += 4 * T) {
    unsigned got[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // the atomics of a batch are in flight together
      const int i = i0 + u * T;
      const unsigned n = i < windows ? count[i] : 0u;
      if (n) got[u] = atomicAdd(fill + (size_t)i * kFillStride, n);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * T;
      if (i < windows && count[i]) count[i] = got[u] - first[i];
    }
  }
  __syncthreads();
  for (unsigned k = threadIdx.x; k < total; k += T) {
    const uint4 r = buf[k];
    const int b = (int)((r.x & ~kHeavy) >> LOGW);
    const unsigned slot = count[b] + k;
    if (slot < (unsigned)Wn::kCap)
      recs[(size_t)b * Wn::kCap + slot] = r;
    else if (slot == (unsigned)Wn::kCap)  // one store per window, not one per entry
      flags[1] = 1u;
  }
}

// Sorts key[0 .. m) by N threads (t = 0 .. N - 1) that `sync` holds together.
// The first step of each size compares mirrored places, so that all steps sort
// upwards and places past m act as +infinity.
template <int N, typename Sync>
__device__ __forceinline__ void bitonic(unsigned long long* key, unsigned m, unsigned t,
                                        const Sync& sync) {
  for (unsigned size = 2; size < 2 * m; size <<= 1) {
    for (unsigned d = size >> 1; d > 0; d >>= 1) {
      sync();
      for (unsigned k = t; k < m; k += N) {
        const unsigned p = d == size >> 1 ? (k ^ (size - 1)) : (k ^ d);
        if (p > k && p < m) {
          const unsigned long long x = key[k], y = key[p];
          if (y < x) {
            key[k] = y;
            key[p] = x;
          }
        }
      }
    }
  }
}

// One CTA per window: its entries by (row, column, position) to the output.
// Also copies its share of the offsets.
template <int LOGW>
__global__ void __launch_bounds__(Win<LOGW>::kThreads, 1)
    window_sort_kernel(const unsigned* __restrict__ fill, const uint4* __restrict__ recs,
                       const float* __restrict__ vin, const uint2* __restrict__ row,
                       long long rows, int32_t* __restrict__ offsets,
                       int32_t* __restrict__ indices, float* __restrict__ values) {
  using Wn = Win<LOGW>;
  constexpr int T = Wn::kThreads, P = Wn::kPer;
  extern __shared__ __align__(16) unsigned char dyn[];
  // an entry's key, column << 32 | position; before: the rows' counts and
  // column ranges; after: the sorted columns and values
  unsigned long long* const key = reinterpret_cast<unsigned long long*>(dyn);
  unsigned* const cnt = reinterpret_cast<unsigned*>(dyn);
  unsigned* const cmin = cnt + Wn::W;
  unsigned* const cmax = cmin + Wn::W;
  int* const out_c = reinterpret_cast<int*>(dyn);
  float* const out_v = reinterpret_cast<float*>(dyn) + Wn::kCap;
  unsigned* const start = reinterpret_cast<unsigned*>(dyn + (size_t)Wn::kCap * 8);  // kCap + 1
  uint2* const large = reinterpret_cast<uint2*>(
      dyn + ((size_t)Wn::kCap * 8 + (Wn::kCap + 1) * 4 + 15) / 16 * 16);  // places sorted apart
  __shared__ unsigned n_large;
  const int t = threadIdx.x, b = blockIdx.x;
  const long long stride = (long long)gridDim.x * T;
  for (long long k = (long long)b * T + t; k <= rows; k += stride) offsets[k] = (int32_t)row[k].x;

  const int n = (int)min(fill[(size_t)b * kFillStride], (unsigned)Wn::kCap);
  unsigned before = 0;
  for (int i = t; i < b; i += T) before += __ldg(fill + (size_t)i * kFillStride);
  unsigned base;  // entries of earlier windows
  cta_exclusive<T>(before, &base);

  int c[P];
  float v[P];
  unsigned es[P], pos[P];  // place in the window << 16 | slot
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int k = i * T + t;
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (k < n) r = __ldcs(recs + (size_t)b * Wn::kCap + k);
    es[i] = r.x & (kHeavy | (unsigned)(Wn::W - 1));
    c[i] = (int)r.y;
    pos[i] = r.z;
    v[i] = __uint_as_float(r.w);
  }
  for (int i = t; i < Wn::W; i += T) {
    cnt[i] = 0u;
    cmin[i] = 0xffffffffu;
    cmax[i] = 0u;
  }
  for (int i = t; i <= Wn::kCap; i += T) start[i] = 0u;
  if (t == 0) n_large = 0u;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (i * T + t >= n || (es[i] & kHeavy)) continue;
    atomicAdd(&cnt[es[i]], 1u);
    atomicMin(&cmin[es[i]], (unsigned)c[i]);
    atomicMax(&cmax[es[i]], (unsigned)c[i]);
  }
  __syncthreads();
  // the place that the column suggests between its row's first and last one:
  // never decreases with the column, each step rounds monotonically
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (i * T + t >= n) continue;
    unsigned p = es[i] & ~kHeavy;
    if (!(es[i] & kHeavy)) {
      const unsigned len = cnt[p], lo = cmin[p], hi = cmax[p];
      const float f = (float)len / ((float)(hi - lo) + 1.f);
      p += min((unsigned)((float)((unsigned)c[i] - lo) * f), len - 1u);
    }
    es[i] = p << 16 | atomicAdd(&start[p], 1u);
  }
  __syncthreads();
  {  // counts -> first slots
    constexpr int PB = P;  // consecutive places per thread
    unsigned m[PB], sum = 0;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      m[i] = start[t * PB + i];
      sum += m[i];
    }
    unsigned total;
    unsigned run = cta_exclusive<T>(sum, &total);
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      start[t * PB + i] = run;
      if (m[i] > (unsigned)kRankMax) large[atomicAdd(&n_large, 1u)] = make_uint2(run, m[i]);
      run += m[i];
    }
    if (t == T - 1) start[Wn::kCap] = run;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (i * T + t >= n) continue;
    es[i] += start[es[i] >> 16];
    key[es[i] & 0xffffu] = (unsigned long long)(unsigned)c[i] << 32 | pos[i];
  }
  __syncthreads();
  // rank among the entries of the same place (the same row)
#pragma unroll
  for (int i = 0; i < P; ++i) {
    pos[i] = 0xffffffffu;  // from here on: the sorted place
    if (i * T + t >= n) continue;
    const unsigned e = es[i] >> 16, lo = start[e], hi = start[e + 1];
    if (hi - lo > (unsigned)kRankMax) continue;
    const unsigned long long mine = key[es[i] & 0xffffu];
    unsigned rank = lo;
    for (unsigned j = lo; j < hi; ++j) rank += key[j] < mine;
    pos[i] = rank;
  }
  __syncthreads();
  // places that many entries share: a bitonic sort each, by a warp, or by the
  // CTA when it is long
  const unsigned nl = n_large;
  for (unsigned q = t >> 5; q < nl; q += T / 32)
    if (large[q].y <= (unsigned)kWarpSort)
      bitonic<32>(key + large[q].x, large[q].y, t & 31, [] { __syncwarp(); });
  for (unsigned q = 0; q < nl; ++q)
    if (large[q].y > (unsigned)kWarpSort)
      bitonic<T>(key + large[q].x, large[q].y, t, [] { __syncthreads(); });
  __syncthreads();
  if (nl) {
    // their entries take what the sort left in their slots
#pragma unroll
    for (int i = 0; i < P; ++i) {
      if (i * T + t >= n || pos[i] != 0xffffffffu) continue;
      const unsigned long long k = key[es[i] & 0xffffu];
      c[i] = (int)(k >> 32);
      v[i] = __ldg(vin + (unsigned)k);
      pos[i] = es[i] & 0xffffu;
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (i * T + t >= n) continue;
    out_c[pos[i]] = c[i];
    out_v[pos[i]] = v[i];
  }
  __syncthreads();
  for (int k = t; k < n; k += T) {
    __stcs(indices + base + k, out_c[k]);
    __stcs(values + base + k, out_v[k]);
  }
}

// The two ways.  A status, and *done = whether the arrays are written.
template <int LOGW>
el_status window_sort(el_workspace* w, const el_coo* coo, int32_t* offsets, int32_t* indices,
                      float* values, cudaStream_t s, int sms, bool* done, bool* checked) {
  using Wn = Win<LOGW>;
  *done = *checked = false;
  const long long nnz = coo->nnz, rows = coo->rows, n = rows + 1;
  const int windows = (int)((nnz + Wn::W - 1) / Wn::W);
  const long long blocks = (n + kScan - 1) / kScan;
  // row length counters, window fills and flags (zeroed together), block
  // sums, rows (start, length), records
  const size_t lbytes = round256((size_t)n * 4),
               fbytes = round256((size_t)(windows + 1) * kFillStride * 4),
               sbytes = round256((size_t)blocks * 4), rbytes = round256((size_t)n * 8);
  const size_t total = lbytes + fbytes + sbytes + rbytes + (size_t)windows * Wn::kCap * 16;
  void* stage = nullptr;
  cudaStream_t cs = nullptr;
  cudaEvent_t ev[4];
  el_status st = workspace_stage(w, total, &stage, &cs, ev);
  if (st == EL_ERR_OUT_OF_MEMORY) {  // the radix sort may still fit
    cudaGetLastError();
    return EL_OK;
  }
  if (st != EL_OK) return st;
  char* p = static_cast<char*>(stage);
  unsigned* len = reinterpret_cast<unsigned*>(p);
  unsigned* flags = reinterpret_cast<unsigned*>(p + lbytes);
  unsigned* fill = flags + kFillStride;
  unsigned* sums = reinterpret_cast<unsigned*>(p + lbytes + fbytes);
  uint2* row = reinterpret_cast<uint2*>(p + lbytes + fbytes + sbytes);
  uint4* recs = reinterpret_cast<uint4*>(p + lbytes + fbytes + sbytes + rbytes);
  cudaError_t e = cudaMemsetAsync(p, 0, lbytes + fbytes, s);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo");
  const unsigned grid = (unsigned)std::min<long long>(
      (nnz + 4 * kCountThreads - 1) / (4 * kCountThreads), (long long)sms * 2);
  if (rows <= kSmallRows)
    count_rows_kernel<true><<<grid, kCountThreads, 0, s>>>(
        coo->row_indices, coo->col_indices, (int)nnz, (unsigned)rows, (unsigned)coo->cols, len, flags);
  else
    count_rows_kernel<false><<<grid, kCountThreads, 0, s>>>(
        coo->row_indices, coo->col_indices, (int)nnz, (unsigned)rows, (unsigned)coo->cols, len, flags);
  const bool summed = blocks > kScanThreads;
  if (blocks > 1) block_sums_kernel<<<(unsigned)blocks, kScanThreads, 0, s>>>(len, n, sums);
  if (summed) scan_sums_kernel<<<1, 1024, 0, s>>>(sums, (int)blocks);
  apply_sums_kernel<<<(unsigned)blocks, kScanThreads, 0, s>>>(len, n, sums, summed, row);
  const int msmem = kMoveTile * 16 + windows * 8;
  e = cudaFuncSetAttribute(move_kernel<LOGW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kMoveTile * 16 + kMaxWindows * 8);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: smem attribute");
  move_kernel<LOGW><<<(unsigned)((nnz + kMoveTile - 1) / kMoveTile), kMoveThreads, msmem, s>>>(
      coo->row_indices, coo->col_indices, coo->values, nnz, rows, coo->cols, row, windows, fill,
      recs, flags);
  e = cudaGetLastError();
  unsigned h[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, flags, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: move");
  if (h[0]) return fail(EL_ERR_MALFORMED_CSR, "COO entry outside %lld x %lld",
                        (long long)coo->rows, (long long)coo->cols);
  *checked = true;
  if (h[1]) return EL_OK;  // a window is full
  e = cudaFuncSetAttribute(window_sort_kernel<LOGW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           Wn::kSmem);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: smem attribute");
  window_sort_kernel<LOGW><<<windows, Wn::kThreads, Wn::kSmem, s>>>(
      fill, recs, coo->values, row, rows, offsets, indices, values);
  *done = true;
  return cuda_status(cudaGetLastError(), "el_csr_from_coo: sort");
}

// `checked`: every entry is known to be in range.
el_status radix_sort(el_workspace* w, const el_coo* coo, int32_t* offsets, int32_t* indices,
                     float* values, cudaStream_t s, int sms, bool checked) {
  const long long nnz = coo->nnz;
  const int cbits = bits_for(coo->cols > 0 ? coo->cols : 1);
  // temporaries in the workspace's staging memory:
  // keys in/out, positions in/out, the bad flag, CUB's temporary storage
  const int end_bit = cbits + bits_for(coo->rows > 0 ? coo->rows : 1);
  size_t cub_bytes = 0;
  cub::DoubleBuffer<unsigned long long> kb(nullptr, nullptr);
  cub::DoubleBuffer<int32_t> pb(nullptr, nullptr);
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, kb, pb, (int)nnz, 0, end_bit, s);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: sort size");
  const size_t kbytes = round256((size_t)nnz * 8), pbytes = round256((size_t)nnz * 4);
  const size_t total = 2 * kbytes + 2 * pbytes + 256 + round256(cub_bytes);
  void* stage = nullptr;
  cudaStream_t cs = nullptr;
  cudaEvent_t ev[4];
  const el_status st = workspace_stage(w, total, &stage, &cs, ev);
  if (st != EL_OK) return st;
  char* p = static_cast<char*>(stage);
  unsigned long long* k0 = reinterpret_cast<unsigned long long*>(p);
  unsigned long long* k1 = reinterpret_cast<unsigned long long*>(p + kbytes);
  int32_t* p0 = reinterpret_cast<int32_t*>(p + 2 * kbytes);
  int32_t* p1 = reinterpret_cast<int32_t*>(p + 2 * kbytes + pbytes);
  unsigned* bad = reinterpret_cast<unsigned*>(p + 2 * kbytes + 2 * pbytes);
  void* tmp = p + 2 * kbytes + 2 * pbytes + 256;

  const unsigned grid = (unsigned)std::min<long long>((nnz + 255) / 256, (long long)sms * 8);
  e = cudaMemsetAsync(bad, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo");
  keys_kernel<<<grid, 256, 0, s>>>(coo->row_indices, coo->col_indices, nnz, coo->rows, coo->cols,
                                   cbits, k0, p0, bad);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: keys");
  unsigned h_bad = 0;
  if (!checked) {
    e = cudaMemcpyAsync(&h_bad, bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: check");
  if (h_bad) return fail(EL_ERR_MALFORMED_CSR, "COO entry outside %lld x %lld",
                         (long long)coo->rows, (long long)coo->cols);
  cub::DoubleBuffer<unsigned long long> keys(k0, k1);
  cub::DoubleBuffer<int32_t> pos(p0, p1);
  size_t tb = round256(cub_bytes);
  e = cub::DeviceRadixSort::SortPairs(tmp, tb, keys, pos, (int)nnz, 0, end_bit, s);
  if (e != cudaSuccess) return cuda_status(e, "el_csr_from_coo: sort");
  gather_kernel<<<grid, 256, 0, s>>>(keys.Current(), pos.Current(), coo->values, nnz, cbits,
                                     indices, values);
  const unsigned ogrid =
      (unsigned)std::min<long long>((coo->rows + 1 + 255) / 256, (long long)sms * 8);
  offsets_kernel<<<ogrid, 256, 0, s>>>(keys.Current(), nnz, coo->rows, cbits, offsets);
  return cuda_status(cudaGetLastError(), "el_csr_from_coo: gather");
}

}  // namespace
}  // namespace el

using namespace el;

extern "C" el_status el_csr_from_coo(el_workspace* ws, const el_coo* coo, int32_t* offsets,
                                     int32_t* indices, float* values, el_stream_t stream) {
  if (!coo) return fail(EL_ERR_NULL_POINTER, "coo is NULL");
  if (coo->rows < 0 || coo->cols < 0 || coo->nnz < 0)
    return fail(EL_ERR_INVALID_ARGUMENT, "negative size");
  if (coo->rows >= (1LL << 31) - 1 || coo->cols >= (1LL << 31) || coo->nnz >= (1LL << 31))
    return fail(EL_ERR_OVERFLOW, "sizes exceed int32");
  if (!offsets) return fail(EL_ERR_NULL_POINTER, "offsets is NULL");
  if (coo->nnz > 0 && (!coo->row_indices || !coo->col_indices || !coo->values || !indices ||
                       !values))
    return fail(EL_ERR_NULL_POINTER, "an array is NULL");
  cudaStream_t s = (cudaStream_t)stream;
  const long long nnz = coo->nnz;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
  const int sms = device_info(device).sm_count;
  if (nnz == 0) {
    e = cudaMemsetAsync(offsets, 0, (size_t)(coo->rows + 1) * sizeof(int32_t), s);
    return cuda_status(e, "el_csr_from_coo: offsets");
  }
  el_workspace* w = nullptr;
  el_status st = workspace_resolve(ws, s, device, &w);
  if (st != EL_OK) return st;
  // The window sort keeps a counter per row, so not for mostly empty rows
  // (its temporaries would outgrow the radix sort's), and one per window in
  // shared memory; below one window the radix sort's single CTA is as fast.
  // Small windows give few entries enough CTAs; large ones keep the move's
  // atomics (entries / 4096 x windows) few: 2M entries 197 us by windows of
  // 2048, 3M 193 us by windows of 8192.
  bool done = false, checked = false;
  if (nnz >= Win<11>::W && coo->rows <= 2 * nnz + (1 << 20) &&
      nnz <= (long long)kMaxWindows * Win<13>::W) {
    st = nnz <= kSmallNnz
             ? window_sort<11>(w, coo, offsets, indices, values, s, sms, &done, &checked)
             : window_sort<13>(w, coo, offsets, indices, values, s, sms, &done, &checked);
    if (st != EL_OK || done) return st;
  }
  return radix_sort(w, coo, offsets, indices, values, s, sms, checked);
}
