// CSR x dense SpMM for sm_100a.
//
// Work split (nnz-balanced):
//   * rows with at most SB_HEAVY_ROW_NNZ entries: one warp per row.  L lanes span a column tile
//     with 128-bit loads of the dense operand, the 32/L lane groups take alternate entries of the
//     row, and a fixed-order shuffle tree adds the groups;
//   * heavier rows (hubs of power-law graphs): cut into segments of SB_HEAVY_ROW_NNZ entries by
//     the row plan; one CTA per segment, one partial sum per warp in shared memory, added in warp
//     order; rows with several segments go through a scratch buffer and a fixed-order finalise.
// The CSR column/value streams are read with coalesced no-allocate loads, one 32-entry chunk per
// warp at a time, and handed to the lanes by shuffles; C is written once with streaming stores.
// Large k is cut into column panels on grid.y, so that one panel of the dense operand stays in
// L2 while all rows pass over it.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"

// floats of the dense operand in flight per lane (32 = 128 bytes measured best on B200: 64 loses
// 25 % on the GCN layers to register pressure, 16 loses 4 % there)
#ifndef SB_SPMM_INFLIGHT
#define SB_SPMM_INFLIGHT 32
#endif

// mean stored entries per row below which a launch takes several rows per warp: 64 where the
// whole warp spans one column tile that covers the operand (128 < k <= 256: four rows per warp
// one after the other), 24 otherwise (narrow tiles, a row per lane group: a 4096-row, 41-per-row,
// 64-column product measured 16 us that way against 10 us with a warp per row; and wide operands
// taken in column panels)
#ifndef SB_SPMM_SHORT_ROW_MEAN
#define SB_SPMM_SHORT_ROW_MEAN 24
#endif
#ifndef SB_SPMM_SHORT_ROW_MEAN_FULL_WARP
#define SB_SPMM_SHORT_ROW_MEAN_FULL_WARP 64
#endif

namespace sb {

constexpr int kWarpsPerCta = 8;

template <typename T>
struct SpmmArgs {
  int m;
  int n;               // rows of B
  int k;
  const int* pos;      // first entry of each row ...
  const int* end;      // ... and the one after its last (pos + 1 unless only part of a row is taken)
  const int* crd;
  const T* val;
  const T* B;
  long long ldb;
  const T* bias;
  int relu;
  T* C;
  long long ldc;
  long long stride_val, stride_b, stride_c;
  int skip_heavy;  // rows longer than SB_HEAVY_ROW_NNZ are left to the heavy kernel
  const int* ent;  // optional entry list: entry p of pos[] is entry ent[p] of crd / val
  int val_compact; // with ent: the value of listed entry p is val[p], not val[ent[p]]
  int accumulate;  // add to the existing contents of C (before bias / ReLU)
  int short_rows;  // many rows of a few dozen entries: several rows per warp
};

// ---- vector access: W elements of T by one load / store instruction (4, 8, 16 or 32 bytes) ----
template <typename T, int W>
struct alignas(W * sizeof(T) < 16 ? W * sizeof(T) : 16) Pack {
  T v[W];
};

template <typename T, int W>
__device__ __forceinline__ Pack<T, W> unpack(const unsigned (&r)[W * sizeof(T) / 4]) {
  Pack<T, W> p;
#pragma unroll
  for (int w = 0; w < W; w++) {
    if constexpr (sizeof(T) == 4) {
      if constexpr (std::is_same<T, float>::value) p.v[w] = __uint_as_float(r[w]);
      else p.v[w] = (T)r[w];
    } else {
      const unsigned long long u = ((unsigned long long)r[2 * w + 1] << 32) | r[2 * w];
      if constexpr (std::is_same<T, double>::value) p.v[w] = __longlong_as_double((long long)u);
      else p.v[w] = (T)u;
    }
  }
  return p;
}
template <typename T, int W>
__device__ __forceinline__ void repack(const Pack<T, W>& p, unsigned (&r)[W * sizeof(T) / 4]) {
#pragma unroll
  for (int w = 0; w < W; w++) {
    if constexpr (sizeof(T) == 4) {
      if constexpr (std::is_same<T, float>::value) r[w] = __float_as_uint(p.v[w]);
      else r[w] = (unsigned)p.v[w];
    } else {
      unsigned long long u;
      if constexpr (std::is_same<T, double>::value) u = (unsigned long long)__double_as_longlong(p.v[w]);
      else u = (unsigned long long)p.v[w];
      r[2 * w] = (unsigned)u;
      r[2 * w + 1] = (unsigned)(u >> 32);
    }
  }
}

// Gather of a dense-operand row slice through the read-only path.  (An L2 evict-last policy on
// these loads was measured on the 4096-column configuration and lost 25 %: left out.)
template <typename T, int W>
__device__ __forceinline__ Pack<T, W> ld_dense(const T* p) {
  constexpr int N = W * (int)sizeof(T) / 4;
  unsigned r[N];
  if constexpr (N == 8)
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "l"(p));
  else if constexpr (N == 4)
    asm volatile("ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "l"(p));
  else if constexpr (N == 2)
    asm volatile("ld.global.nc.v2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "l"(p));
  else
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(r[0]) : "l"(p));
  return unpack<T, W>(r);
}

// Present contents of an output slice, or a segment sum another CTA left in L2: not through L1.
// ONCE: read once and rewritten, marked for early eviction.
template <typename T, int W, bool ONCE = false>
__device__ __forceinline__ Pack<T, W> ld_l2(const T* p) {
  constexpr int N = W * (int)sizeof(T) / 4;
  unsigned r[N];
  const unsigned* q = reinterpret_cast<const unsigned*>(p);
  if constexpr (N >= 4) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const uint4* s = reinterpret_cast<const uint4*>(q + i);
      const uint4 x = ONCE ? __ldcs(s) : __ldcg(s);
      r[i] = x.x; r[i + 1] = x.y; r[i + 2] = x.z; r[i + 3] = x.w;
    }
  } else if constexpr (N == 2) {
    const uint2* s = reinterpret_cast<const uint2*>(q);
    const uint2 x = ONCE ? __ldcs(s) : __ldcg(s);
    r[0] = x.x; r[1] = x.y;
  } else {
    r[0] = ONCE ? __ldcs(q) : __ldcg(q);
  }
  return unpack<T, W>(r);
}

// Streaming (evict-first) store of an output slice: written once, never re-read here.
template <typename T, int W>
__device__ __forceinline__ void st_stream(T* p, const Pack<T, W>& x) {
  constexpr int N = W * (int)sizeof(T) / 4;
  unsigned r[N];
  repack<T, W>(x, r);
  if constexpr (N == 8)
    asm volatile("st.global.cs.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
  else if constexpr (N == 4)
    asm volatile("st.global.cs.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3])
                 : "memory");
  else if constexpr (N == 2)
    asm volatile("st.global.cs.v2.b32 [%0], {%1,%2};" ::"l"(p), "r"(r[0]), "r"(r[1]) : "memory");
  else
    asm volatile("st.global.cs.b32 [%0], %1;" ::"l"(p), "r"(r[0]) : "memory");
}

// Plain store of a slice in scratch.
template <typename T, int W>
__device__ __forceinline__ void store_plain(T* p, const Pack<T, W>& x) {
#pragma unroll
  for (int w = 0; w < W; w++) p[w] = x.v[w];
}

__device__ __forceinline__ double ld_stream(const double* p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_stream(const unsigned* p) {
  return (unsigned)ld_stream(reinterpret_cast<const int*>(p));
}
__device__ __forceinline__ unsigned long long ld_stream(const unsigned long long* p) {
  return (unsigned long long)__double_as_longlong(ld_stream(reinterpret_cast<const double*>(p)));
}

template <typename T>
__device__ __forceinline__ T mul_add(T a, T b, T c) {
  if constexpr (std::is_same<T, float>::value) return fmaf(a, b, c);
  else if constexpr (std::is_same<T, double>::value) return fma(a, b, c);
  else return a * b + c;
}

// Row pitch of the dense operand in elements: 32 bits, but for the one-element form, which takes
// any layout (the 64-bit product costs two more instructions per entry).
template <int W>
using Pitch = typename std::conditional<W == 1, unsigned long long, unsigned>::type;

// Accumulate entries [b, e) of one row into acc[] for this lane's columns.
// L lanes per group (each lane VEC packs of W elements, pack v at column (l + v*L)*W of the tile),
// G = 32/L groups; group g takes entries b+g, b+g+G, ...  EXACT: the tile has no ragged edge.
template <typename T, int L, int VEC, int W, bool EXACT>
__device__ __forceinline__ void accumulate_range(Pack<T, W> (&acc)[VEC], const int* __restrict__ crd,
                                                 const T* __restrict__ val,
                                                 const T* __restrict__ Bcol, Pitch<W> ldb,
                                                 int b, int e, int lane, const bool (&col_ok)[VEC],
                                                 const int* __restrict__ ent = nullptr,
                                                 bool val_compact = false, bool have_first = false,
                                                 int first_j = 0, T first_a = T(0)) {
  constexpr int G = 32 / L;
  constexpr int STEPS = 32 / G;
  // entries in flight per lane: SB_SPMM_INFLIGHT floats' worth of gathered operand, rounded down
  // to a power of two (it divides STEPS)
  constexpr int UMAX = SB_SPMM_INFLIGHT * 4 / (VEC * W * (int)sizeof(T));
  constexpr int UP = UMAX >= 32 ? 32 : UMAX >= 16 ? 16 : UMAX >= 8 ? 8 : UMAX >= 4 ? 4 : UMAX >= 2 ? 2 : 1;
  constexpr int U = (STEPS < UP) ? STEPS : UP;
  const int g = lane / L;
  // software pipeline: the next chunk's indices/values are in flight while this chunk's rows of
  // the dense operand are gathered (the caller may have fetched the first chunk already)
  int next_j = first_j;
  T next_a = first_a;
  if (!have_first && b + lane < e) {
    const int x = ent ? ld_stream(ent + b + lane) : b + lane;
    next_j = ld_stream(crd + x);
    next_a = ld_stream(val + (val_compact ? b + lane : x));
  }
  for (int p0 = b; p0 < e; p0 += 32) {
    const int cnt = min(32, e - p0);
    const int my_j = next_j;
    const T my_a = next_a;
    if (p0 + 32 + lane < e) {
      const int x = ent ? ld_stream(ent + p0 + 32 + lane) : p0 + 32 + lane;
      next_j = ld_stream(crd + x);
      next_a = ld_stream(val + (val_compact ? p0 + 32 + lane : x));
    }
    if (cnt == 32) {
#pragma unroll 1
      for (int s0 = 0; s0 < STEPS; s0 += U) {
        T a[U];
        Pack<T, W> bv[U][VEC];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int t = (s0 + u) * G + g;
          const unsigned j = (unsigned)__shfl_sync(FULL, my_j, t);
          a[u] = __shfl_sync(FULL, my_a, t);
          const T* brow = Bcol + (size_t)((unsigned long long)j * ldb);
#pragma unroll
          for (int v = 0; v < VEC; v++) {
            if (EXACT || col_ok[v]) {
              bv[u][v] = ld_dense<T, W>(brow + v * L * W);
            } else {
#pragma unroll
              for (int w = 0; w < W; w++) bv[u][v].v[w] = T(0);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
          for (int v = 0; v < VEC; v++) {
#pragma unroll
            for (int w = 0; w < W; w++) acc[v].v[w] = mul_add(a[u], bv[u][v].v[w], acc[v].v[w]);
          }
        }
      }
    } else {
      // the row's last, part-filled chunk: UT entries per lane group in flight (one at a time for
      // full 1 KB slices, where a batch was measured slower: registers)
      constexpr int UT = (VEC * W * (int)sizeof(T) >= 32 && L == 32) ? 1 : (U < 4 ? U : 4);
#pragma unroll 1
      for (int t0 = 0; t0 < cnt; t0 += G * UT) {
        T a[UT];
        Pack<T, W> bv[UT][VEC];
#pragma unroll
        for (int u = 0; u < UT; u++) {
          const int t = t0 + u * G + g;
          const unsigned j = (unsigned)__shfl_sync(FULL, my_j, t & 31);
          a[u] = __shfl_sync(FULL, my_a, t & 31);
          const bool in = t < cnt;
          if (!in) a[u] = T(0);
          const T* brow = Bcol + (size_t)((unsigned long long)j * ldb);
#pragma unroll
          for (int v = 0; v < VEC; v++) {
            if (in && (EXACT || col_ok[v])) {
              bv[u][v] = ld_dense<T, W>(brow + v * L * W);
            } else {
#pragma unroll
              for (int w = 0; w < W; w++) bv[u][v].v[w] = T(0);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < UT; u++) {
#pragma unroll
          for (int v = 0; v < VEC; v++) {
#pragma unroll
            for (int w = 0; w < W; w++) acc[v].v[w] = mul_add(a[u], bv[u][v].v[w], acc[v].v[w]);
          }
        }
      }
    }
  }
}

template <typename T, int L, int VEC, int W>
__device__ __forceinline__ void reduce_groups(Pack<T, W> (&acc)[VEC]) {
#pragma unroll
  for (int o = L; o < 32; o <<= 1) {
#pragma unroll
    for (int v = 0; v < VEC; v++) {
#pragma unroll
      for (int w = 0; w < W; w++) acc[v].v[w] += __shfl_xor_sync(FULL, acc[v].v[w], o);
    }
  }
}

template <typename T, int W>
__device__ __forceinline__ Pack<T, W> epilogue(Pack<T, W> s, const T* bias, int col, int relu) {
  if (bias) {
    const Pack<T, W> bb = ld_dense<T, W>(bias + col);
#pragma unroll
    for (int w = 0; w < W; w++) s.v[w] += bb.v[w];
  }
  if (relu) {
#pragma unroll
    for (int w = 0; w < W; w++) s.v[w] = s.v[w] > T(0) ? s.v[w] : T(0);
  }
  return s;
}

template <typename T, int VEC, int W>
__device__ __forceinline__ void zero_acc(Pack<T, W> (&acc)[VEC]) {
#pragma unroll
  for (int v = 0; v < VEC; v++) {
#pragma unroll
    for (int w = 0; w < W; w++) acc[v].v[w] = T(0);
  }
}

// The sums of one row, or of a segment of it, over the whole CTA: a slice of [b, e) per warp (a
// multiple of 32 entries), the warps' sums added in warp order by warp 0, whose first L lanes hold
// the result.
template <typename T, int L, int VEC, int W, bool EXACT>
__device__ __forceinline__ void cta_range(Pack<T, W> (&s)[VEC], Pack<T, W> (&part)[kWarpsPerCta][VEC][L],
                                          const SpmmArgs<T>& a, const T* val, const T* Bcol, int b, int e,
                                          const bool (&col_ok)[VEC]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane % L;
  const int slice = (((e - b) + 32 * kWarpsPerCta - 1) / (32 * kWarpsPerCta)) * 32;
  const int wb = min(e, b + warp * slice), we = min(e, wb + slice);
  zero_acc<T, VEC, W>(s);
  accumulate_range<T, L, VEC, W, EXACT>(s, a.crd, val, Bcol, (Pitch<W>)a.ldb, wb, we, lane, col_ok, a.ent,
                                        a.val_compact != 0);
  reduce_groups<T, L, VEC, W>(s);
  if (lane < L) {
#pragma unroll
    for (int v = 0; v < VEC; v++) part[warp][v][l] = s[v];
  }
  __syncthreads();
  if (warp == 0 && lane < L) {
#pragma unroll
    for (int v = 0; v < VEC; v++) {
      s[v] = part[0][v][l];
#pragma unroll
      for (int w2 = 1; w2 < kWarpsPerCta; w2++) {
        const Pack<T, W> t = part[w2][v][l];
#pragma unroll
        for (int w = 0; w < W; w++) s[v].v[w] += t.v[w];
      }
    }
  }
}

// One warp per R consecutive rows; grid = (row blocks, column tiles, batch).  R = 1 in general;
// launches over many short rows (the entries a block plan leaves outside its blocks) use R = 4:
// the rows' bounds and first index chunks are fetched together, so the rows share one start-up
// latency instead of paying it each.
constexpr int kShortRowsPerWarp = 4;  // (2 and 8 measured slower)
// (four CTAs per SM for the short-row form: 64 registers; five and three measured slower.  The
// forms with narrower loads hold more addresses and spill at 64: three.)
template <typename T, int VEC, int W>
constexpr int kShortRowCtas = (std::is_same<T, float>::value && W >= 4) ? 4 : 3;
template <typename T, int L, int VEC, int W, bool EXACT, int R>
__device__ __forceinline__ void rows_body(const SpmmArgs<T>& a, int block_x) {
  constexpr int TILE = L * W * VEC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row_base = (block_x * kWarpsPerCta + warp) * R;
  if (row_base >= a.m) return;
  const long long bz = blockIdx.z;
  const int l = lane % L;
  const int col0 = blockIdx.y * TILE + l * W;
  const T* val = a.val + bz * a.stride_val;
  bool col_ok[VEC];
#pragma unroll
  for (int v = 0; v < VEC; v++) col_ok[v] = EXACT || (col0 + v * L * W) < a.k;
  int pb = 0, pe = 0;  // lane r < R: bounds of row row_base + r (rows past the end: empty)
  if (lane < R && row_base + lane < a.m) {
    pb = __ldg(a.pos + row_base + lane);
    pe = __ldg(a.end + row_base + lane);
  }
  int first_j[R];
  T first_a[R];
  if (R > 1) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int b = __shfl_sync(FULL, pb, r), e = __shfl_sync(FULL, pe, r);
      first_j[r] = 0;
      first_a[r] = T(0);
      if (b + lane < e) {
        const int x = a.ent ? ld_stream(a.ent + b + lane) : b + lane;
        first_j[r] = ld_stream(a.crd + x);
        first_a[r] = ld_stream(val + (a.val_compact ? b + lane : x));
      }
    }
  }
#pragma unroll 1
  for (int rr = 0; rr < R; rr++) {
    const int row = row_base + rr;
    if (row >= a.m) break;
    const int b = __shfl_sync(FULL, pb, rr), e = __shfl_sync(FULL, pe, rr);
    if (a.skip_heavy && e - b > SB_HEAVY_ROW_NNZ) continue;
    Pack<T, W> acc[VEC];
    zero_acc<T, VEC, W>(acc);
    T* crow = a.C + bz * a.stride_c + (long long)row * a.ldc;
    if (a.accumulate && lane < L) {
      // the row's present contents start the first lane group's sums: the load overlaps the
      // index loads and gathers instead of sitting between the reduction and the store
#pragma unroll
      for (int v = 0; v < VEC; v++) {
        if (col_ok[v]) acc[v] = ld_l2<T, W>(crow + col0 + v * L * W);
      }
    }
    int fj = 0;
    T fa = T(0);
    if (R > 1) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (r == rr) { fj = first_j[r]; fa = first_a[r]; }
      }
    }
    accumulate_range<T, L, VEC, W, EXACT>(acc, a.crd, val, a.B + bz * a.stride_b + col0, (Pitch<W>)a.ldb,
                                          b, e, lane, col_ok, a.ent, a.val_compact != 0, R > 1, fj, fa);
    reduce_groups<T, L, VEC, W>(acc);
    if (lane < L) {
#pragma unroll
      for (int v = 0; v < VEC; v++) {
        const int col = col0 + v * L * W;
        if (!col_ok[v]) continue;
        st_stream<T, W>(crow + col, epilogue<T, W>(acc[v], a.bias, col, a.relu));
      }
    }
  }
}

template <typename T, int L, int VEC, int W, bool EXACT, int R>
__global__ void __launch_bounds__(kWarpsPerCta * 32, R > 1 ? kShortRowCtas<T, VEC, W> : 1)
spmm_rows_kernel(SpmmArgs<T> a) {
  rows_body<T, L, VEC, W, EXACT, R>(a, (int)blockIdx.x);
}

// Short rows, narrow tiles (L <= 16 lanes span the tile): each of the 32/L lane groups of a warp
// takes a row of its own, so a warp works on 32/L rows at once and no sums cross lanes.  A group
// reads its row's indices/values L at a time and keeps SB_SPMM_INFLIGHT floats of gathered
// operand rows in flight per lane.  Rows longer than kGroupedMaxRow (but not heavy) are done by
// the whole warp afterwards, like the general kernel does.
#ifndef SB_SPMM_GROUPED_MAX_ROW
#define SB_SPMM_GROUPED_MAX_ROW 64
#endif
constexpr int kGroupedMaxRow = SB_SPMM_GROUPED_MAX_ROW;

template <typename T, int L, int W, bool EXACT>
__device__ __forceinline__ void rows_grouped_body(const SpmmArgs<T>& a, int block_x) {
  constexpr int G = 32 / L;
  constexpr int TILE = L * W;
  constexpr int UMAX = SB_SPMM_INFLIGHT * 4 / (W * (int)sizeof(T));
  constexpr int U = (L < UMAX) ? L : UMAX;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row_base = (block_x * kWarpsPerCta + warp) * G;
  if (row_base >= a.m) return;
  const int g = lane / L, l = lane % L;
  const int row = row_base + g;
  const long long bz = blockIdx.z;
  const T* val = a.val + bz * a.stride_val;
  const int col0 = blockIdx.y * TILE + l * W;
  const bool col_ok = EXACT || col0 < a.k;
  const T* Bcol = a.B + bz * a.stride_b + col0;
  const Pitch<W> ldb = (Pitch<W>)a.ldb;
  int b = 0, e = 0;
  if (row < a.m) {
    b = __ldg(a.pos + row);
    e = __ldg(a.end + row);
  }
  const bool heavy = a.skip_heavy && (e - b) > SB_HEAVY_ROW_NNZ;
  const bool by_warp = !heavy && (e - b) > kGroupedMaxRow;
  const bool mine = row < a.m && !heavy && !by_warp;
  const int ge = mine ? e : b;
  T* crow = a.C + bz * a.stride_c + (long long)row * a.ldc;
  Pack<T, W> acc;
#pragma unroll
  for (int w = 0; w < W; w++) acc.v[w] = T(0);
  if (a.accumulate && mine && col_ok) acc = ld_l2<T, W>(crow + col0);
  const int longest = __reduce_max_sync(FULL, ge - b);
  int next_j = 0;
  T next_a = T(0);
  if (b + l < ge) {
    const int x = a.ent ? ld_stream(a.ent + b + l) : b + l;
    next_j = ld_stream(a.crd + x);
    next_a = ld_stream(val + (a.val_compact ? b + l : x));
  }
#pragma unroll 1
  for (int q0 = 0; q0 < longest; q0 += L) {
    const int p0 = b + q0;
    const int my_j = next_j;
    const T my_a = next_a;
    if (p0 + L + l < ge) {
      const int x = a.ent ? ld_stream(a.ent + p0 + L + l) : p0 + L + l;
      next_j = ld_stream(a.crd + x);
      next_a = ld_stream(val + (a.val_compact ? p0 + L + l : x));
    }
    const int cnt = ge - p0;                    // entries this group still has (may be <= 0)
    const int most = min(L, longest - q0);      // warp-uniform
#pragma unroll 1
    for (int t0 = 0; t0 < most; t0 += U) {
      T av[U];
      Pack<T, W> bv[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int t = t0 + u;
        const unsigned j = (unsigned)__shfl_sync(FULL, my_j, t, L);
        av[u] = __shfl_sync(FULL, my_a, t, L);
        if (t < cnt && col_ok) {
          bv[u] = ld_dense<T, W>(Bcol + (size_t)((unsigned long long)j * ldb));
        } else {
          av[u] = T(0);
#pragma unroll
          for (int w = 0; w < W; w++) bv[u].v[w] = T(0);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int w = 0; w < W; w++) acc.v[w] = mul_add(av[u], bv[u].v[w], acc.v[w]);
      }
    }
  }
  if (mine && col_ok) st_stream<T, W>(crow + col0, epilogue<T, W>(acc, a.bias, col0, a.relu));
  // rows too long for one lane group: the whole warp, one row after the other
  if (__any_sync(FULL, by_warp)) {
#pragma unroll 1
    for (int gg = 0; gg < G; gg++) {
      if (!__shfl_sync(FULL, (int)by_warp, gg * L)) continue;
      const int rb = __shfl_sync(FULL, b, gg * L), re = __shfl_sync(FULL, e, gg * L);
      Pack<T, W> acc2[1];
      bool ok2[1] = {col_ok};
      zero_acc<T, 1, W>(acc2);
      T* crow2 = a.C + bz * a.stride_c + (long long)(row_base + gg) * a.ldc;
      if (a.accumulate && lane < L && col_ok) acc2[0] = ld_l2<T, W>(crow2 + col0);
      accumulate_range<T, L, 1, W, EXACT>(acc2, a.crd, val, Bcol, ldb, rb, re, lane, ok2, a.ent,
                                          a.val_compact != 0);
      reduce_groups<T, L, 1, W>(acc2);
      if (lane < L && col_ok) st_stream<T, W>(crow2 + col0, epilogue<T, W>(acc2[0], a.bias, col0, a.relu));
    }
  }
}

template <typename T, int L, int W, bool EXACT>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4)
spmm_rows_grouped_kernel(SpmmArgs<T> a) {
  rows_grouped_body<T, L, W, EXACT>(a, (int)blockIdx.x);
}

template <typename T>
struct HeavyArgs {
  const int* hdr;
  const int* heavy_row;
  const int* heavy_seg0;
  const int* heavy_nseg;
  const int* seg_heavy;
  T* scratch;                // [batch][segments][k] segment sums of multi-segment rows
  long long scratch_batch;   // elements between batch items
  int* arrived;              // [batch][column tiles][segments] segments done per heavy row (zeroed)
  int segments;              // slots per arrival counter row (>= the plan's segment count)
  int first_heavy;           // blockIdx.x of the first heavy CTA; the row CTAs take the other indices
};

// One CTA per heavy-row segment.  The CTA that finishes a row's last outstanding segment adds
// the row's segment sums in segment order and writes the row (fixed order, whichever CTA does it).
template <typename T, int L, int VEC, int W, bool EXACT>
__device__ __forceinline__ void heavy_body(const SpmmArgs<T>& a, const HeavyArgs<T>& h, int seg) {
  constexpr int TILE = L * W * VEC;
  __shared__ Pack<T, W> part[kWarpsPerCta][VEC][L];
  __shared__ int s_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = __ldg(h.seg_heavy + seg);
  const int row = __ldg(h.heavy_row + slot);
  const int seg0 = __ldg(h.heavy_seg0 + slot);
  const int nseg = __ldg(h.heavy_nseg + slot);
  const int rb = __ldg(a.pos + row), re = __ldg(a.end + row);
  const int sb_ = rb + (seg - seg0) * SB_HEAVY_ROW_NNZ;
  const int se = min(re, sb_ + SB_HEAVY_ROW_NNZ);
  const long long bz = blockIdx.z;
  const int l = lane % L;
  const int col0 = blockIdx.y * TILE + l * W;
  bool col_ok[VEC];
#pragma unroll
  for (int v = 0; v < VEC; v++) col_ok[v] = EXACT || (col0 + v * L * W) < a.k;
  Pack<T, W> s[VEC];
  cta_range<T, L, VEC, W, EXACT>(s, part, a, a.val + bz * a.stride_val, a.B + bz * a.stride_b + col0, sb_, se,
                                 col_ok);
  if (warp == 0 && lane < L) {
#pragma unroll
    for (int v = 0; v < VEC; v++) {
      const int col = col0 + v * L * W;
      if (!col_ok[v]) continue;
      if (nseg == 1) {
        T* dst = a.C + bz * a.stride_c + (long long)row * a.ldc + col;
        if (a.accumulate) {
          const Pack<T, W> old = ld_l2<T, W>(dst);
#pragma unroll
          for (int w = 0; w < W; w++) s[v].v[w] += old.v[w];
        }
        st_stream<T, W>(dst, epilogue<T, W>(s[v], a.bias, col, a.relu));
      } else {
        T* dst = h.scratch + bz * h.scratch_batch + (long long)seg * a.k + col;
#pragma unroll
        for (int w = 0; w < W; w++) dst[w] = s[v].v[w];
        __threadfence();  // the segment sum is visible before this CTA counts itself done
      }
    }
  }
  if (nseg == 1) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    int* cnt = h.arrived + ((long long)bz * gridDim.y + blockIdx.y) * h.segments + seg0;
    s_last = (atomicAdd(cnt, 1) == nseg - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const T* src = h.scratch + bz * h.scratch_batch + (long long)seg0 * a.k;
  T* crow = a.C + bz * a.stride_c + (long long)row * a.ldc;
  const int tile0 = blockIdx.y * TILE;
  for (int c = threadIdx.x; c < TILE; c += blockDim.x) {
    const int col = tile0 + c;
    if (col >= a.k) break;
    Pack<T, 1> x;
    x.v[0] = a.accumulate ? __ldcg(crow + col) : T(0);
    for (int t = 0; t < nseg; t++) x.v[0] += __ldcg(src + (long long)t * a.k + col);
    st_stream<T, 1>(crow + col, epilogue<T, 1>(x, a.bias, col, a.relu));
  }
}

// The segments of all heavy rows; grid.x CTAs take them in turn (one each when the host knows
// their number).
template <typename T, int L, int VEC, int W, bool EXACT>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
spmm_heavy_kernel(SpmmArgs<T> a, HeavyArgs<T> h) {
  const int n = __ldg(h.hdr + 1);
  for (int seg = blockIdx.x; seg < n; seg += gridDim.x) {
    heavy_body<T, L, VEC, W, EXACT>(a, h, seg);
    __syncthreads();   // the shared buffers are written again
  }
}

// Rows and heavy-row segments in one launch; grid = (row blocks + segments, column tiles, batch):
// the segment CTAs [first_heavy, first_heavy + segments) run beside the row CTAs instead of
// waiting for a launch of their own.
// (Both bodies inlined want 76-96 registers; three CTAs per SM, like the rows kernel alone gets,
// caps that at 85.)
template <typename T, int L, int VEC, int W, bool EXACT, int R>
__global__ void __launch_bounds__(kWarpsPerCta * 32, R > 1 ? 4 : 3)
spmm_rows_heavy_kernel(SpmmArgs<T> a, HeavyArgs<T> h) {
  const int hb = (int)blockIdx.x - h.first_heavy;
  if (hb >= 0 && hb < h.segments) {
    if (hb < __ldg(h.hdr + 1)) heavy_body<T, L, VEC, W, EXACT>(a, h, hb);
  } else {
    rows_body<T, L, VEC, W, EXACT, R>(a, hb < 0 ? (int)blockIdx.x : hb - h.segments + h.first_heavy);
  }
}

template <typename T, int L, int W, bool EXACT>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4)
spmm_grouped_heavy_kernel(SpmmArgs<T> a, HeavyArgs<T> h) {
  const int hb = (int)blockIdx.x - h.first_heavy;
  if (hb >= 0 && hb < h.segments) {
    if (hb < __ldg(h.hdr + 1)) heavy_body<T, L, 1, W, EXACT>(a, h, hb);
  } else {
    rows_grouped_body<T, L, W, EXACT>(a, hb < 0 ? (int)blockIdx.x : hb - h.segments + h.first_heavy);
  }
}

template <typename T, int L, int VEC, int W, bool EXACT>
static int launch_vec2(const SpmmArgs<T>& a, int64_t batch, const void* plan, int64_t nnz,
                       int64_t plan_segments, void* scratch, cudaStream_t st) {
  constexpr int TILE = L * W * VEC;
  constexpr int THREADS = kWarpsPerCta * 32;
  const unsigned tiles = (unsigned)ceil_div(a.k, TILE);
  if (tiles > 65535)
    return fail(SB_ERR_UNSUPPORTED, "spmm: at most %lld columns with this layout, got %d", 65535ll * TILE, a.k);
  // short rows: a row per lane group where the tile is narrow, else several rows per warp
  constexpr bool kGrouped = (L <= 16 && VEC == 1);
  const int rows_per_warp = !a.short_rows ? 1 : (kGrouped ? 32 / L : kShortRowsPerWarp);
  const int64_t row_ctas = ceil_div(ceil_div(a.m, rows_per_warp), kWarpsPerCta);
  dim3 grid((unsigned)row_ctas, tiles, (unsigned)batch);
  if constexpr (std::is_same<T, float>::value) if (plan && plan_segments != 0) {
    PlanView pv = plan_view(plan, nnz);
    const int64_t segs = plan_segments < 0 ? pv.cap_seg : plan_segments;
    T* sums = static_cast<T*>(scratch);
    int* arrived = reinterpret_cast<int*>(sums + (size_t)segs * a.k * batch);
    HeavyArgs<T> h{pv.hdr, pv.heavy_row, pv.heavy_seg0, pv.heavy_nseg, pv.seg_heavy,
                   sums, (long long)segs * a.k, arrived, (int)segs, 0};
    SB_CUDA(cudaMemsetAsync(arrived, 0, (size_t)segs * tiles * batch * sizeof(int), st));
    // Long rows: the rows in a launch of their own, then the segments (one launch with both
    // bodies needs 10-20 more registers per thread and measured 3 % / 20 % slower at 256 / 64
    // columns on a 2 M-row power-law graph).  Short-row passes (a row chunk's share of a
    // matrix: few segments, a launch of their own would leave most SMs idle): one launch, the
    // segment CTAs behind the row CTAs (4 % faster than in front at 256 columns).
    if (!a.short_rows) {
      spmm_rows_kernel<T, L, VEC, W, EXACT, 1><<<grid, THREADS, 0, st>>>(a);
      SB_LAUNCH_CHECK("spmm_rows_kernel");
      spmm_heavy_kernel<T, L, VEC, W, EXACT><<<dim3((unsigned)segs, tiles, (unsigned)batch), THREADS, 0, st>>>(a, h);
      SB_LAUNCH_CHECK("spmm_heavy_kernel");
      return SB_OK;
    }
    h.first_heavy = (int)row_ctas;
    dim3 both((unsigned)(segs + row_ctas), tiles, (unsigned)batch);
    if constexpr (kGrouped) spmm_grouped_heavy_kernel<T, L, W, EXACT><<<both, THREADS, 0, st>>>(a, h);
    else spmm_rows_heavy_kernel<T, L, VEC, W, EXACT, kShortRowsPerWarp><<<both, THREADS, 0, st>>>(a, h);
    SB_LAUNCH_CHECK("spmm_rows_heavy_kernel");
    return SB_OK;
  }
  if (!a.short_rows) spmm_rows_kernel<T, L, VEC, W, EXACT, 1><<<grid, THREADS, 0, st>>>(a);
  else if constexpr (kGrouped) spmm_rows_grouped_kernel<T, L, W, EXACT><<<grid, THREADS, 0, st>>>(a);
  else spmm_rows_kernel<T, L, VEC, W, EXACT, kShortRowsPerWarp><<<grid, THREADS, 0, st>>>(a);
  SB_LAUNCH_CHECK("spmm_rows_kernel");
  return SB_OK;
}

// Launch for one element type and load width; SB_GO picks the kernel form, SB_GO_FIT its variant
// without a ragged column edge where the tile divides the width.
// (entry tiles when the caller gave their workspace; they have one variant for both)
#define SB_GO(L, VEC, W, EXACT)                                                                \
  do {                                                                                         \
    if (tile_ws && a.ldb * (long long)sizeof(T) < (1ll << 32))                                 \
      return launch_tiles<T, L, VEC, W>(a, nnz, tile_ws, st);                                  \
    return launch_vec2<T, L, VEC, W, EXACT>(a, batch, plan, nnz, plan_segments, scratch, st);  \
  } while (0)
#define SB_GO_FIT(L, VEC, W)                                  \
  do {                                                        \
    if (a.k % ((L) * (VEC) * (W)) == 0) SB_GO(L, VEC, W, true); \
    SB_GO(L, VEC, W, false);                                  \
  } while (0)

// Largest power of two, at most 32, that every row slice of B and C (and the bias) is aligned to.
template <typename T>
inline unsigned spmm_alignment(const SpmmArgs<T>& a) {
  const unsigned long long bits = 32u | reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C) |
                                  reinterpret_cast<uintptr_t>(a.bias) |
                                  (sizeof(T) * (unsigned long long)(a.ldb | a.ldc | a.stride_b | a.stride_c | a.k));
  return (unsigned)(bits & (~bits + 1));
}

// Defined in spmm.cu (16 and 32 byte loads), spmm_f32_narrow.cu and spmm_typed.cu.
int spmm_dispatch_f32(const SpmmArgs<float>& a, int64_t batch, const void* plan, int64_t nnz,
                      int64_t plan_segments, void* scratch, void* tile_ws, cudaStream_t st);
int spmm_dispatch_f32_narrow(const SpmmArgs<float>& a, int64_t batch, const void* plan, int64_t nnz,
                             int64_t plan_segments, void* scratch, void* tile_ws, cudaStream_t st);
template <typename T>
int spmm_dispatch_typed(const SpmmArgs<T>& a, int64_t nnz, void* tile_ws, cudaStream_t st);

}  // namespace sb
