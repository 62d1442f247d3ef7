// Sorting kernels of the SpGEMM (see spgemm.cu): one output row, or one bucket of a long row, per
// warp or CTA.
//
// The products of a row are expanded into shared memory, each with a key (column, ordinal of the
// product) in one 32- or 64-bit word, and the keys are sorted in registers by a bitonic network
// (R keys per thread; strides below R inside the thread, then shuffles, then shared memory).  Equal
// columns are then neighbours in the order of their ordinals: a run is summed in that order, so the
// result has the same bits on every run without atomics, and the values move once (they are looked
// up by ordinal).  Hash tables with 64-bit atomics, a compaction and a sort of key-value pairs did
// the same at 5.8 G products/s.
// Bound: the gather of B's rows (12 entries each on a power-law matrix: two or three sectors per
// row and array) and the issue rate of the network: about 2 instructions per key and 512-key row.
#pragma once

#include <limits.h>

#include <type_traits>

#include "common.cuh"

namespace sb {

typedef unsigned long long Slot;   // bits of a product: double for the float types, else the integer

template <typename T>
constexpr bool kIsFloat = std::is_same<T, float>::value || std::is_same<T, double>::value;

template <typename T>
__device__ __forceinline__ Slot product_bits(T a, T b) {
  if constexpr (kIsFloat<T>) return (Slot)__double_as_longlong((double)a * (double)b);
  else return (Slot)(T)(a * b);
}

struct CsrIn {
  const int* Apos; const int* Acrd; const void* Aval;
  const int* Bpos; const int* Bcrd; const void* Bval;
};

// Sum of a run of products in a fixed order.  float: the products are exact in double.  double:
// the rounding errors of the additions are carried along (two-sum), as exact as the 64-bit
// fixed-point sums of the long rows.
template <typename T>
struct RunSum {
  double s = 0.0, c = 0.0;
  T i = T(0);
  __device__ __forceinline__ void add(Slot bits) {
    if constexpr (std::is_same<T, float>::value) {
      s += __longlong_as_double((long long)bits);
    } else if constexpr (std::is_same<T, double>::value) {
      const double x = __longlong_as_double((long long)bits), t = s + x, z = t - s;
      c += (s - (t - z)) + (x - z);
      s = t;
    } else {
      i += (T)bits;
    }
  }
  __device__ __forceinline__ T value() const {
    if constexpr (std::is_same<T, float>::value) return (float)s;
    else if constexpr (std::is_same<T, double>::value) return fabs(s) <= 1.7976931348623157e308 ? s + c : s;
    else return i;
  }
};

// ---- bitonic network ---------------------------------------------------------------------------
// Ascending sort of NT * R keys, thread t holding elements t * R .. t * R + R - 1.  `xch`: NT * R
// keys of shared memory (used when the CTA has more than one warp).
// (Only the steps inside a thread are unrolled: the register file is indexed by constants, and the
// loops over sizes and thread distances keep the code small.)
template <typename KEY, int R>
__device__ __forceinline__ void compare_inside(KEY (&k)[R], int stride, bool up) {
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int j = i ^ stride;
    if (j > i) {
      const KEY lo = k[i] < k[j] ? k[i] : k[j], hi = k[i] < k[j] ? k[j] : k[i];
      k[i] = up ? lo : hi;
      k[j] = up ? hi : lo;
    }
  }
}

template <typename KEY, int R, int NT>
__device__ __forceinline__ void bitonic_sort(KEY (&k)[R], KEY* xch, int tid) {
  // sizes up to R / 2: the direction depends on the place inside the thread
#pragma unroll
  for (int size = 2; size < R; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int j = i ^ stride;
        if (j > i) {
          const KEY lo = k[i] < k[j] ? k[i] : k[j], hi = k[i] < k[j] ? k[j] : k[i];
          k[i] = (i & size) == 0 ? lo : hi;
          k[j] = (i & size) == 0 ? hi : lo;
        }
      }
    }
  }
  // sizes R, 2 R, ...: `span` threads are merged
#pragma unroll 1
  for (int span = 1; span <= NT; span <<= 1) {
    const bool up = (tid & span) == 0;
#pragma unroll 1
    for (int ts = span >> 1; ts > 0; ts >>= 1) {
      const bool keep_min = up == ((tid & ts) == 0);
      if (NT == 32 || ts < 32) {
#pragma unroll
        for (int i = 0; i < R; i++) {
          const KEY o = __shfl_xor_sync(FULL, k[i], ts);
          k[i] = (k[i] < o) == keep_min ? k[i] : o;
        }
      } else {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < R; i++) xch[i * NT + tid] = k[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < R; i++) {
          const KEY o = xch[i * NT + (tid ^ ts)];
          k[i] = (k[i] < o) == keep_min ? k[i] : o;
        }
      }
    }
#pragma unroll
    for (int stride = R >> 1; stride > 0; stride >>= 1) compare_inside<KEY, R>(k, stride, up);
  }
}

template <int NT>
__device__ __forceinline__ void group_sync() {
  if (NT == 32) __syncwarp(); else __syncthreads();
}

// Sorts the first `count` <= NT * R keys of `keys` in place (groups of several warps use the rest of
// the NT * R slots as well).
template <typename KEY, int R, int NT>
__device__ __forceinline__ void sort_keys(KEY* keys, int count, int tid) {
  KEY k[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int e = tid + i * NT;      // (any assignment will do: the keys are in no order yet)
    k[i] = e < count ? keys[e] : ~KEY(0);
  }
  bitonic_sort<KEY, R, NT>(k, keys, tid);
  group_sync<NT>();
#pragma unroll
  for (int i = 0; i < R; i++)
    if (tid * R + i < count) keys[tid * R + i] = k[i];
  group_sync<NT>();
}

// ---- emission -------------------------------------------------------------------------------------
// Distinct columns (key >> shift) among the sorted keys [b, e) of a row that begins at keys[0]: their
// number, a warp together.
template <typename KEY>
__device__ __forceinline__ int count_runs(const KEY* keys, int b, int e, int shift, int lane) {
  int heads = 0;
  for (int x0 = b; x0 < e; x0 += 32) {
    const int x = x0 + lane;
    const bool head = x < e && (x == 0 || (keys[x] >> shift) != (keys[x - 1] >> shift));
    heads += __popc(__ballot_sync(FULL, head));
  }
  return heads;
}
// ... and for each one write(o, column, first, last): o = at, at + 1, ..., [first, last) its run of
// sorted keys (which may end behind e, at most at `count`).  Returns their number.
template <typename KEY, typename F>
__device__ __forceinline__ int write_runs(const KEY* keys, int b, int e, int count, int shift, int lane, int col0,
                                          long long at, F&& write) {
  int n = 0;
  for (int x0 = b; x0 < e; x0 += 32) {
    const int x = x0 + lane;
    const KEY col = x < e ? keys[x] >> shift : KEY(0);
    const bool head = x < e && (x == 0 || col != (keys[x - 1] >> shift));
    const unsigned heads = __ballot_sync(FULL, head);
    if (head) {
      // up to the next head, or, from the last one of the 32, as far as the column goes
      const unsigned next = heads >> lane >> 1;
      int last = next ? x + __ffs(next) : min(e, x0 + 32);
      if (!next)
        while (last < count && (keys[last] >> shift) == col) last++;
      write(at + n + __popc(heads & ((1u << lane) - 1u)), col0 + (int)col, x, last);
    }
    n += __popc(heads);
  }
  return n;
}
// Both for a group of NT threads, every warp a contiguous part (s_part: one int per warp); returns
// the number of distinct columns.
template <typename KEY, int NT, bool EMIT, typename F>
__device__ __forceinline__ int emit_runs(const KEY* keys, int count, int shift, int tid, int* s_part, int col0,
                                         long long base, F&& write) {
  constexpr int NW = NT / 32;
  const int warp = tid >> 5, lane = tid & 31;
  const int per = NW == 1 ? count : ((count + NT - 1) / NT) * 32;
  const int b = NW == 1 ? 0 : min(count, warp * per), e = NW == 1 ? count : min(count, b + per);
  int before = 0, total = 0;
  if (NW > 1 || !EMIT) {
    total = count_runs<KEY>(keys, b, e, shift, lane);
    if (NW > 1) {
      if (lane == 0) s_part[warp] = total;
      __syncthreads();
      total = 0;
#pragma unroll
      for (int w = 0; w < NW; w++) {
        const int h = s_part[w];
        if (w < warp) before += h;
        total += h;
      }
    }
  }
  if (EMIT) {
    const int n = write_runs<KEY>(keys, b, e, count, shift, lane, col0, base + before, write);
    if (NW == 1) total = n;
  }
  return total;
}

// ---- expansion ------------------------------------------------------------------------------------
// The products of `entries` A entries from pa0 on (at most 32, one per lane) spread evenly over the lanes
// of a warp: lane l looks up the B row of entry pa0 + l, a warp scan of the row lengths numbers
// the products, and every lane then takes products lane, lane + 32, ... — a 5-step search over
// the scanned lengths tells which entry a product belongs to.  No lane idles on a short B row and
// the index loads of 32 entries are in flight together, instead of one dependent chain
// (A entry -> B row pointers -> B entries) per entry.  `emit(ordinal, a_value, pb)` is called once
// per product with its number in this group, the value of its A entry (T(0) in the symbolic phase)
// and its position in B; the number of products is returned.
template <typename T, bool NUMERIC, typename F>
__device__ __forceinline__ int expand_products(const CsrIn& in, int pa0, int entries, int lane, F&& emit) {
  int bb = 0, len = 0;
  T a = T(0);
  if (lane < entries) {
    const int pa = pa0 + lane;
    const int j = __ldg(in.Acrd + pa);
    bb = __ldg(in.Bpos + j);
    len = __ldg(in.Bpos + j + 1) - bb;
    if (NUMERIC) a = static_cast<const T*>(in.Aval)[pa];
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  const int excl = incl - len;
#pragma unroll 4
  for (int q0 = 0; q0 < total; q0 += 32) {
    const int q = q0 + lane;
    // largest e with excl[e] <= q (lanes past the end search too: shuffles need the whole warp)
    int e = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int v = __shfl_sync(FULL, excl, e + step);
      if (v <= q) e += step;
    }
    const int off = __shfl_sync(FULL, bb - excl, e);
    const T e_a = NUMERIC ? __shfl_sync(FULL, a, e) : T(0);
    if (q < total) emit(q, e_a, off + q);
  }
  return total;
}

// The same for a CTA of NT threads, NT entries at a time: product q goes to thread q % NT whatever the
// lengths of the B rows are, the search runs over the scanned lengths in shared memory.  (With a
// warp per 32 entries, a row whose products come mostly from one long B row - the usual long row of
// a power-law matrix - kept one warp busy and the rest waiting.)  `part` of `parts` CTAs takes every
// parts-th NT products.
template <typename T, int NT>
struct ExpandSmem {
  int excl[NT], off[NT];
  T a[NT];
  int part[NT / 32];
};
// `turn(first, total, find)` is called per NT entries, with the number of the first product and of products; find(q)
// = entry of the turn's product q.
template <typename T, bool NUMERIC, int NT, typename F>
__device__ __forceinline__ void expand_turns(const CsrIn& in, int ab, int ae, ExpandSmem<T, NT>& sm, int tid,
                                             F&& turn) {
  const int warp = tid >> 5, lane = tid & 31;
  // (unsigned: what is looked at ahead of A's last entries, up to 2^31 - 1 of them, lies beyond an int)
  const unsigned a0 = ab, a1 = ae;
  int first = 0;
  // (groups of 512 threads and more, which rows of several NT entries come to: the row pointers of the next NT
  // entries and the columns of the NT after those are on their way meanwhile; the others mostly take one turn)
  constexpr bool AHEAD = NT >= 512;
  int next_bb = 0, next_len = 0, next_j = 0;
  T next_a = T(0);
  auto fetch_row = [&](unsigned pa, int j) {
    next_bb = next_len = 0;
    if (pa < a1) {
      if (!AHEAD) j = __ldg(in.Acrd + pa);
      next_bb = __ldg(in.Bpos + j);
      next_len = __ldg(in.Bpos + j + 1) - next_bb;
      if (NUMERIC) next_a = static_cast<const T*>(in.Aval)[pa];
    }
  };
  auto fetch_column = [&](unsigned pa) {
    if (pa < a1) next_j = __ldg(in.Acrd + pa);
  };
  if constexpr (AHEAD) {
    fetch_column(a0 + tid);
    const int j = next_j;
    fetch_column(a0 + NT + tid);
    fetch_row(a0 + tid, j);
  }
  for (unsigned p0 = a0; p0 < a1; p0 += NT) {
    if (!AHEAD) fetch_row(p0 + tid, 0);
    const int bb = next_bb, len = next_len;
    if (NUMERIC) sm.a[tid] = next_a;
    if (AHEAD && p0 + NT < a1) {
      fetch_row(p0 + NT + tid, next_j);
      fetch_column(p0 + 2 * NT + tid);
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sm.part[warp] = incl;
    __syncthreads();
    int excl = incl - len, total = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++) {
      const int c = sm.part[w];
      if (w < warp) excl += c;
      total += c;
    }
    sm.excl[tid] = excl;
    sm.off[tid] = bb - excl;
    __syncthreads();
    turn(first, total, [&](int q) {
      int e = 0;   // largest e with excl[e] <= q
#pragma unroll
      for (int step = NT / 2; step > 0; step >>= 1)
        if (sm.excl[e + step] <= q) e += step;
      return e;
    });
    first += total;
    __syncthreads();
  }
}

template <typename T, bool NUMERIC, int NT, typename F>
__device__ __forceinline__ void expand_cta(const CsrIn& in, int ab, int ae, ExpandSmem<T, NT>& sm, int tid, F&& emit,
                                           int part = 0, int parts = 1) {
  expand_turns<T, NUMERIC, NT>(in, ab, ae, sm, tid, [&](int first, int total, auto&& find) {
#pragma unroll 4
    for (unsigned u = part * NT + tid; u < (unsigned)total; u += parts * NT) {
      const int q = (int)u, e = find(q);
      emit(first + q, NUMERIC ? sm.a[e] : T(0), sm.off[e] + q);
    }
  });
}

// All products of A row [ab, ae) to shared memory: keys[o] = column << shift | o, prods[o]; their
// number is known beforehand.  One warp (`sm` unused) or a CTA.  COLUMNS: keys[o] = column alone.
template <typename T, bool NUMERIC, typename KEY, int NT, bool COLUMNS = false>
__device__ __forceinline__ void expand_row(const CsrIn& in, int ab, int ae, int shift, KEY* keys, Slot* prods,
                                           int tid, ExpandSmem<T, NT>* sm) {
  const T* Bval = static_cast<const T*>(in.Bval);
  auto put = [&](int o, T a, int pb) {
    const KEY c = (KEY)(unsigned)__ldg(in.Bcrd + pb);
    keys[o] = COLUMNS ? c : (c << shift) | (KEY)o;
    if (NUMERIC) prods[o] = product_bits<T>(a, __ldg(Bval + pb));
  };
  if constexpr (NT == 32) {
    int first = 0;
    for (int left = ae - ab; left > 0; left -= 32)
      first += expand_products<T, NUMERIC>(in, ae - left, min(left, 32), tid, [&](int o, T a, int pb) {
        put(first + o, a, pb);
      });
    __syncwarp();
  } else {
    expand_cta<T, NUMERIC, NT>(in, ab, ae, *sm, tid, put);
  }
}

// The kernels of the bins run side by side: each lets the next launch begin at its own start and ends
// only after the launch before it (its last CTA waits for that; the others free their places), so that
// what follows the last one follows all of them.
__device__ __forceinline__ void let_next_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void end_after_previous() {
  if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

struct RowsOut {
  int* row_cnt;         // distinct columns per row (null: not wanted)
  const int* off;       // [row] where the row's entries go (numeric)
  int* crd;
  void* val;
};

template <typename T, bool NUMERIC, typename KEY, int R, int NT>
__device__ __forceinline__ int sort_and_emit(KEY* keys, const Slot* prods, int count, int shift, int tid, int* s_part,
                                             long long base, const RowsOut& out) {
  sort_keys<KEY, R, NT>(keys, count, tid);
  T* val = static_cast<T*>(out.val);
  const KEY mask = ((KEY)1 << shift) - 1;
  return emit_runs<KEY, NT, NUMERIC>(keys, count, shift, tid, s_part, 0, base,
                                     [&](long long o, int col, int x, int last) {
    out.crd[o] = col;
    RunSum<T> s;
    for (; x < last; x++) s.add(prods[(int)(keys[x] & mask)]);
    val[o] = s.value();
  });
}

// Rows of at most 128 products: a warp each, the network as long as the row needs.
constexpr int kWarpCap = 128;
template <typename T, bool NUMERIC, typename KEY, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
spgemm_warp_kernel(const int* __restrict__ rows, int nrows, const int* __restrict__ upper, CsrIn in, int shift,
                   RowsOut out) {
  __shared__ KEY s_keys[WARPS][kWarpCap];
  __shared__ Slot s_prods[WARPS][NUMERIC ? kWarpCap : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * WARPS + warp;
  let_next_begin();
  if (r >= nrows) {
    end_after_previous();
    return;
  }
  const int i = __ldg(rows + r);
  const int count = __ldg(upper + i), ab = __ldg(in.Apos + i), ae = __ldg(in.Apos + i + 1);
  const long long base = NUMERIC ? __ldg(out.off + i) : 0;
  KEY* keys = s_keys[warp];
  Slot* prods = s_prods[warp];
  expand_row<T, NUMERIC, KEY, 32>(in, ab, ae, shift, keys, prods, lane, nullptr);
  int u;
#define SB_SORT(R) u = sort_and_emit<T, NUMERIC, KEY, R, 32>(keys, prods, count, shift, lane, nullptr, base, out)
  if (count <= 32) SB_SORT(1);
  else if (count <= 64) SB_SORT(2);
  else SB_SORT(4);
#undef SB_SORT
  if (out.row_cnt && lane == 0) out.row_cnt[i] = u;
  end_after_previous();
}

// Rows of at most RMAX NT products: a CTA of NT threads each.  (A single warp for 129 to 512
// products took 57 ns per thousand products, serial in its slabs of A entries.)
template <typename T, bool NUMERIC, typename KEY, int NT, int RMAX>
__global__ void __launch_bounds__(NT)
spgemm_cta_kernel(const int* __restrict__ rows, const int* __restrict__ upper, CsrIn in, int shift, RowsOut out) {
  constexpr int CAP = RMAX * NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Slot* prods = reinterpret_cast<Slot*>(smem_raw);
  KEY* keys = reinterpret_cast<KEY*>(smem_raw + (NUMERIC ? sizeof(Slot) * CAP : 0));
  __shared__ ExpandSmem<T, NT> s_expand;
  int* s_part = s_expand.part;
  let_next_begin();
  const int i = __ldg(rows + blockIdx.x), tid = threadIdx.x;
  const int count = __ldg(upper + i), ab = __ldg(in.Apos + i), ae = __ldg(in.Apos + i + 1);
  const long long base = NUMERIC ? __ldg(out.off + i) : 0;
  expand_row<T, NUMERIC, KEY, NT>(in, ab, ae, shift, keys, prods, tid, &s_expand);
  int u;
  if (count <= RMAX / 2 * NT)
    u = sort_and_emit<T, NUMERIC, KEY, RMAX / 2, NT>(keys, prods, count, shift, tid, s_part, base, out);
  else
    u = sort_and_emit<T, NUMERIC, KEY, RMAX, NT>(keys, prods, count, shift, tid, s_part, base, out);
  if (out.row_cnt && tid == 0) out.row_cnt[i] = u;
  end_after_previous();
}

// Rows of 2049 to 8192 products: a CTA each, the row's columns cut into segments of equal width that a
// warp sorts each.  The network over the whole row would need 64-bit keys (21 bits of column and 13 of
// ordinal on a 2 M-column matrix), 128 KB of shared memory and ten exchanges through it: 4.6 ms
// for 10,562 rows where the segments take 1.0 ms.  Segments of more than 512 products (columns
// crowded together) are sorted by the CTA in shared memory.
// Bound: the network's issue rate and the emission's chains.  16 warps and 32 segments a row, two rows per SM; where
// there are no more rows than SMs 32 warps and 64 segments (a row of 7,700 products and 1,500 entries: 50 us, 31 so).
// (Ranks by counting within some 4,000 buckets in place of the networks of all the CTA kernels took fewer
// instructions in ALU and more waiting: 1.15 ms to 1.44 for the 56,789 rows of 513 to 2048 products.)
constexpr int kSplitCap = 8192, kSegmentSort = 512, kSplitOrd = 13;
template <int NT>
constexpr int kSplitSegments = NT / 16;

// Ascending sort of any number of keys in shared memory by NT threads: the bitonic network in the form
// in which every comparison puts the smaller key first, so that places behind the end need no key.
template <typename KEY, int NT>
__device__ __noinline__ void sort_in_smem(KEY* keys, int count, int tid) {
  for (int size = 2; size < 2 * count; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const int flip = stride == size >> 1 ? size - 1 : stride;
      __syncthreads();
      for (int x = tid; x < count; x += NT) {
        const int y = x ^ flip;
        if (y > x && y < count && keys[y] < keys[x]) {
          const KEY t = keys[x];
          keys[x] = keys[y];
          keys[y] = t;
        }
      }
    }
  }
  __syncthreads();
}

// Segment of a column: column / width (width = columns / segments, rounded up; scale = 2^32 / width, rounded up:
// at most one too many).
__device__ __forceinline__ int segment_of(unsigned col, int width, unsigned scale) {
  const int seg = width > 1 ? (int)__umulhi(col, scale) : (int)col;
  return seg - ((unsigned)seg * (unsigned)width > col);
}
// Exclusive sums of the segments' counts by a warp, the total behind them (known to lane 31).
template <int SEGMENTS>
__device__ __forceinline__ int exclusive_segments(const int* cnt, int* start, int lane) {
  constexpr int PER = SEGMENTS / 32;
  int c[PER], incl = 0;
#pragma unroll
  for (int q = 0; q < PER; q++) incl += c[q] = cnt[PER * lane + q];
  int at = -incl;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  at += incl;
#pragma unroll
  for (int q = 0; q < PER; q++) {
    start[PER * lane + q] = at;
    at += c[q];
  }
  if (lane == 31) start[SEGMENTS] = incl;
  return incl;
}

template <typename T, bool NUMERIC, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
spgemm_split_kernel(const int* __restrict__ rows, const int* __restrict__ upper, CsrIn in, int width, unsigned scale,
                    RowsOut out) {
  constexpr int NW = NT / 32, R = kSplitCap / NT, kSegments = kSplitSegments<NT>;
  typedef unsigned KEY;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Slot* prods = reinterpret_cast<Slot*>(smem_raw);
  KEY* keys = reinterpret_cast<KEY*>(smem_raw + (NUMERIC ? sizeof(Slot) * kSplitCap : 0));
  __shared__ ExpandSmem<T, NT> s_expand;
  __shared__ int s_cnt[kSegments + 1], s_start[kSegments + 1], s_u[kSegments];
  const int i = __ldg(rows + blockIdx.x), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int count = __ldg(upper + i), ab = __ldg(in.Apos + i), ae = __ldg(in.Apos + i + 1);
  const long long base = NUMERIC ? __ldg(out.off + i) : 0;
  let_next_begin();
  if (tid < kSegments) s_cnt[tid] = 0;
  expand_row<T, NUMERIC, KEY, NT, true>(in, ab, ae, 0, keys, prods, tid, &s_expand);
  // columns to their segments (in any order: the sort brings it), the ordinal below the column
  KEY c[R];
  int place[R];                // segment << 16 | place in it
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int x = tid + q * NT;
    if (x < count) {
      const int seg = segment_of(keys[x], width, scale);
      c[q] = keys[x] - (unsigned)(seg * width);
      place[q] = seg << 16 | atomicAdd(&s_cnt[seg], 1);
    }
  }
  __syncthreads();
  if (warp == 0) exclusive_segments<kSegments>(s_cnt, s_start, lane);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int x = tid + q * NT;
    if (x < count) keys[s_start[place[q] >> 16] + (place[q] & 0xffff)] = c[q] << kSplitOrd | (KEY)x;
  }
  __syncthreads();
  for (int seg = 0; seg < kSegments; seg++) {
    const int n = s_start[seg + 1] - s_start[seg];
    if (n > kSegmentSort) sort_in_smem<KEY, NT>(keys + s_start[seg], n, tid);
  }
  for (int seg = warp; seg < kSegments; seg += NW) {
    const int b = s_start[seg], n = s_start[seg + 1] - b;
    if (n <= kSegmentSort) {
      if (n > 256) sort_keys<KEY, 16, 32>(keys + b, n, lane);
      else if (n > 128) sort_keys<KEY, 8, 32>(keys + b, n, lane);
      else if (n > 64) sort_keys<KEY, 4, 32>(keys + b, n, lane);
      else if (n > 32) sort_keys<KEY, 2, 32>(keys + b, n, lane);
      else if (n > 1) sort_keys<KEY, 1, 32>(keys + b, n, lane);
    }
    const int u = count_runs<KEY>(keys + b, 0, n, kSplitOrd, lane);
    if (lane == 0) s_u[seg] = u;
  }
  __syncthreads();
  if (warp == 0) {
    const int u = exclusive_segments<kSegments>(s_u, s_cnt, lane);
    if (out.row_cnt && lane == 31) out.row_cnt[i] = u;
  }
  if (NUMERIC) {
    __syncthreads();
    T* val = static_cast<T*>(out.val);
    for (int seg = warp; seg < kSegments; seg += NW) {
      const int b = s_start[seg], n = s_start[seg + 1] - b;
      const KEY* k = keys + b;
      write_runs<KEY>(k, 0, n, n, kSplitOrd, lane, seg * width, base + s_cnt[seg],
                      [&](long long o, int col, int x, int last) {
        out.crd[o] = col;
        RunSum<T> s;
        for (; x < last; x++) s.add(prods[(int)(k[x] & (kSplitCap - 1))]);
        val[o] = s.value();
      });
    }
  }
  end_after_previous();
}

}  // namespace sb
