// SpMM over tiles of stored entries: the form for one matrix, with no row plan.
//
// What it is for: rows of very different lengths (power-law matrices) and short rows.  With a warp
// or lane group per row, most of the GPU waits for the few that got long rows.  Here a CTA takes
// the rows that begin in a window of TE consecutive entries, so every CTA has about the same number
// of entries, and inside it a row is taken by whatever suits its length:
//   up to kGroupRow entries    one lane group (L lanes across the operand's columns), rows of similar
//                              length side by side in a warp
//   up to kWarpRow             the lane groups of a warp, a slice each
//   longer                     all lane groups of the CTA, in units of kUnit entries; the unit sums
//                              of a row of several units are added by a second launch, every eighth
//                              one in order, then these eight sums (it also writes the rows without
//                              entries)
// Nothing is built beforehand and no host decision depends on the matrix.  Which sums are formed in
// which order depends on a row's own length only, not on where the row lies: the same bits on every
// run, and for a block of rows the same as for the whole matrix.
// The window's indices and values go to shared memory by cp.async while the first row is looked
// for; gathers keep U operand rows per lane group in flight.
// Bound: L2 -> SM gathers of operand rows (17 TB/s measured for random rows of 64 bytes and more)
// where the operand stays in L2, else DRAM on the gathers.
#pragma once

#include "spmm_kernels.cuh"

namespace sb {

constexpr int kTileThreadsMm = 256;
constexpr int kTileWarps = kTileThreadsMm / 32;
constexpr int kUnit = 512;             // a window's last row or unit reaches up to this far behind it
// Largest window.  Wide rows (L = 32) have work enough in 1536 entries and lose residency to more
// (6 M entries, 256 columns: 371 us, 415 with 3072; 2048 saves uniform matrices of 0.9 to 1.2 M entries a second
// wave, 64.4 us to 60.7 with 256 columns, but leaves a power law's windows uneven, 64.8 to 67.5 with 77); narrow
// ones gain by having their start-up spread over twice as many (0.8 M entries in rows of 8, 64 columns: 27.0 us, 22.9
// with 3072).
// 8-byte types, whose entries take 16 bytes: as much as lets three CTAs stay within 196 KB of shared memory.
// Beyond that 23 KB are left to L1 in place of 55 and the gathers wait for it (120,000 rows of 27 entries, the same
// operands over and over: 16 float64 columns 47.0 us with 3072, 42.7 with this, 3 columns 41.5, 34.5).
constexpr int tile_window(int L, int size = 4) { return L == 32 ? 1536 : size == 8 ? 2560 : 3072; }
// Rows of up to this length go to a lane group.  32 lets the warp's other groups help with a row of
// a power-law graph (2 M rows, 64 columns: 6.10 ms with 64, 5.66 with 32); the 8 groups of four
// lanes have too little of a 33-entry row each (the same 16 float64 columns: 46.6 us with 32, 42.7 with 40, 43.1
// with 64; power law of mean 20, 8 columns: 27.6, 28.0, 30.0).
template <int L>
constexpr int kGroupRow = L == 4 ? 40 : 32;
constexpr int kWarpRow = 192;
constexpr int kTileRowCap = 1024;      // row pointers kept in shared memory at a time
// Rows of a window that a warp takes, and units that the CTA takes, at most.
template <int L, int SIZE>
constexpr int kWarpList = tile_window(L, SIZE) / (kGroupRow<L> + 1) + 2;
template <int L, int SIZE>
constexpr int kUnitList = tile_window(L, SIZE) / kWarpRow + tile_window(L, SIZE) / kUnit + 4;
// Classes of similar length among the rows that a lane group takes.  A warp's groups take rows of one class,
// the longest first: in the order of the matrix they waited for the longest of their 2 to 8 rows.  (GCN
// layer of 2 M rows, 202 M entries, 64-column panels: 20.4 ms in the matrix's order, 19.1 by class; power law
// of mean 12, 32 columns: 46.8 us, 39.8; 60,000 rows of 16, 7 columns: 15.0, 13.1.  Taken as one stream of entries
// per group across the rows' ends, an operand row fetched for every one added, the same rows took 1.7 to 2 times as
// long.)
constexpr int kShortClasses = 4;

// Resident CTAs per SM the kernels are compiled for (64 / 80 registers; measured per lane count).
constexpr int tile_ctas(int L) { return L == 32 ? 4 : 3; }
// Entries per window, a multiple of 32: as few full waves of CTAs over the chip as windows of at
// most tile_window(L) allow (a last wave that is half empty costs as much as a full one), at least 64
// and at least four per lane group.
inline int tile_entries(int64_t nnz, int L, int size) {
  const int64_t slots = (int64_t)sm_count() * tile_ctas(L);
  const int64_t waves = std::max<int64_t>(1, ceil_div(nnz, slots * tile_window(L, size)));
  const int64_t te = ceil_div(ceil_div(nnz, slots * waves), 32) * 32;
  return (int)std::min<int64_t>(std::max<int64_t>(te, std::max(64, 1024 / L)), tile_window(L, size));
}

template <typename T>
struct TileArgs {
  int nnz, entries, tiles, panels;
  T* first;         // [nnz / kUnit + 1][k] sums of the first units of rows of several units ...
  T* rest;          // ... and of their other units; index = first entry of the unit / kUnit
};

// One stored entry in shared memory, read by one load.
template <typename T>
struct alignas(sizeof(T) == 4 ? 8 : 16) Entry {
  T a;
  int j;
};

struct TileUnit {
  int row, begin, len, whole;   // whole: the row has no other unit
};

template <typename T, int L, int VEC, int W>
struct TileSmem {
  Pack<T, W> part[kTileWarps][VEC][L];
  Entry<T> entry[tile_window(L, sizeof(T)) + kUnit];
  int pos[kTileRowCap + 2];
  TileUnit by_warp[kWarpList<L, sizeof(T)>], by_cta[kUnitList<L, sizeof(T)>];
  // rows of a turn that a lane group takes, by length (where a warp has several groups)
  // (two classes share an array, one from each end)
  unsigned short short_row[kShortClasses / 2][L == 32 ? 1 : kTileRowCap];
  int n_short[kShortClasses];
  int n_warp, n_cta, next_warp, next_row;
  int count[kTileWarps];
};

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, uint64_t policy) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(BYTES), "l"(policy)
               : "memory");
}

template <typename T, int L, int VEC, int W>
__device__ __forceinline__ void tile_store_row(const SpmmArgs<T>& a, int row, int col0, const bool (&col_ok)[VEC],
                                               const Pack<T, W> (&sum)[VEC]) {
  T* crow = a.C + (long long)row * a.ldc;
#pragma unroll
  for (int v = 0; v < VEC; v++) {
    const int col = col0 + v * L * W;
    if (col_ok[v]) st_stream<T, W>(crow + col, epilogue<T, W>(sum[v], a.bias, col, a.relu));
  }
}

// Initial sums of the lane group that will store the row: zero, or the row's present contents
// (accumulation), loaded here so that they arrive with the first gathers.
template <typename T, int L, int VEC, int W>
__device__ __forceinline__ void tile_begin_row(Pack<T, W> (&s)[VEC], const SpmmArgs<T>& a, int row, int col0,
                                               const bool (&col_ok)[VEC], bool owner) {
  zero_acc<T, VEC, W>(s);
  if (!a.accumulate || !owner) return;
  const T* crow = a.C + (long long)row * a.ldc;
#pragma unroll
  for (int v = 0; v < VEC; v++)
    if (col_ok[v]) s[v] = ld_l2<T, W, true>(crow + col0 + v * L * W);
}

// acc += the entries [b, e) of the window, one after the other, U operand rows in flight.  Lanes
// beyond the last column read the first one's slice (`Bcol` points there) and drop the result.
template <typename T, int VEC, int W, int U>
__device__ __forceinline__ void tile_add(Pack<T, W> (&acc)[VEC], const Entry<T>* entry, int b, int e,
                                         const char* const (&Bcol)[VEC], unsigned pitch) {
  int p = b;
#pragma unroll 1
  for (; p + U <= e; p += U) {
    Entry<T> x[U];
    Pack<T, W> bv[U][VEC];
#pragma unroll
    for (int u = 0; u < U; u++) {
      x[u] = entry[p + u];
#pragma unroll
      for (int v = 0; v < VEC; v++)
        bv[u][v] = ld_dense<T, W>(reinterpret_cast<const T*>(Bcol[v] + (unsigned long long)(unsigned)x[u].j * pitch));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
#pragma unroll
      for (int v = 0; v < VEC; v++) {
#pragma unroll
        for (int w = 0; w < W; w++) acc[v].v[w] = mul_add(x[u].a, bv[u][v].v[w], acc[v].v[w]);
      }
    }
  }
  if (p < e) {
    Entry<T> x[U];
    Pack<T, W> bv[U][VEC];
#pragma unroll
    for (int u = 0; u + 1 < U; u++) {
      x[u].a = T(0);
      if (p + u < e) {
        x[u] = entry[p + u];
#pragma unroll
        for (int v = 0; v < VEC; v++)
          bv[u][v] =
              ld_dense<T, W>(reinterpret_cast<const T*>(Bcol[v] + (unsigned long long)(unsigned)x[u].j * pitch));
      } else {
#pragma unroll
        for (int v = 0; v < VEC; v++) {
#pragma unroll
          for (int w = 0; w < W; w++) bv[u][v].v[w] = T(0);
        }
      }
    }
#pragma unroll
    for (int u = 0; u + 1 < U; u++) {
#pragma unroll
      for (int v = 0; v < VEC; v++) {
#pragma unroll
        for (int w = 0; w < W; w++) acc[v].v[w] = mul_add(x[u].a, bv[u][v].v[w], acc[v].v[w]);
      }
    }
  }
}

template <typename T, int L, int VEC, int W>
__global__ void __launch_bounds__(kTileThreadsMm, tile_ctas(L))
spmm_tile_kernel(SpmmArgs<T> a, TileArgs<T> t) {
  using Smem = TileSmem<T, L, VEC, W>;
  constexpr int G = 32 / L, NG = kTileWarps * G;
  constexpr int UMAX = SB_SPMM_INFLIGHT * 4 / (VEC * W * (int)sizeof(T));
  constexpr int U = UMAX >= 8 ? 8 : UMAX >= 4 ? 4 : 2;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane % L, g = lane / L;
  const unsigned pitch = (unsigned)(a.ldb * (long long)sizeof(T));
  // (set up while the kernel before it still runs; the operands may be that kernel's results)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int e0 = (int)blockIdx.x * t.entries, e1 = min(t.nnz, e0 + t.entries);
  const int staged = min(t.nnz, e1 + kUnit) - e0;
  // (read once: marked for early eviction, the operand's rows are what L2 should keep)
  uint64_t once;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
  for (int i = tid; i < staged; i += kTileThreadsMm) {
    cp_async<4>(&sm.entry[i].j, a.crd + e0 + i, once);
    cp_async<(int)sizeof(T)>(&sm.entry[i].a, a.val + e0 + i, once);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");

  // rows in turns of kTileRowCap, from the one that holds the first entry not dealt with
  for (int next = e0; next < e1;) {
    const int r0 = cta_row_of<kTileThreadsMm>(a.pos, a.m, next, sm.count);
    for (int i = tid; i < kTileRowCap + 1; i += kTileThreadsMm) sm.pos[i] = __ldg(a.pos + min(a.m, r0 + i));
    if (tid < kShortClasses) sm.n_short[tid] = 0;
    if (tid == 0) sm.n_warp = sm.n_cta = sm.next_warp = sm.next_row = 0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // rows and units too long for a lane group, as far as they begin in the window
    int rows = 0;                        // rows of this turn that begin before e1
    for (int i = tid; i < kTileRowCap; i += kTileThreadsMm) {
      const int b = sm.pos[i], len = sm.pos[i + 1] - b;
      const bool here = b < e1 && r0 + i < a.m;
      rows += here;
      if constexpr (G > 1) {
        if (!__any_sync(FULL, here)) break;
        const int c = here && b >= next && len > 0 && len <= kGroupRow<L>
                          ? kShortClasses - 1 - (len - 1) / (kGroupRow<L> / kShortClasses) : -1;
        unsigned mine = 0, lanes = 0;    // lanes of this lane's class, of class `lane`
#pragma unroll
        for (int q = 0; q < kShortClasses; q++) {
          const unsigned x = __ballot_sync(FULL, c == q);
          mine = c == q ? x : mine;
          lanes = lane == q ? x : lanes;
        }
        int at = 0;
        if (lane < kShortClasses) at = atomicAdd(&sm.n_short[lane], __popc(lanes));
        at = __shfl_sync(FULL, at, c & (kShortClasses - 1)) + __popc(mine & ((1u << lane) - 1u));
        if (c >= 0) sm.short_row[c >> 1][c & 1 ? kTileRowCap - 1 - at : at] = (unsigned short)i;
      }
      if (!here || len <= kGroupRow<L>) continue;
      if (len <= kWarpRow) {
        if (b >= next) sm.by_warp[atomicAdd(&sm.n_warp, 1)] = TileUnit{r0 + i, b, len, 1};
      } else {
        // (first unit at or behind the window's start; a row that began before a later turn's first
        // entry was dealt with by the turn before)
        int u = b >= next ? 0 : (next == e0 ? (e0 - b + kUnit - 1) / kUnit : INT32_MAX / kUnit);
        for (; u < (len + kUnit - 1) / kUnit && b + u * kUnit < e1; u++)
          sm.by_cta[atomicAdd(&sm.n_cta, 1)] =
              TileUnit{r0 + i, b + u * kUnit, min(kUnit, len - u * kUnit), len <= kUnit};
      }
    }
    int n_short[kShortClasses];          // (rows up to the class's end)
    if constexpr (G > 1) {
      __syncthreads();
      rows = 0;
#pragma unroll
      for (int c = 0; c < kShortClasses; c++) n_short[c] = rows += sm.n_short[c];
    } else {
      rows = __reduce_add_sync(FULL, rows);
      if (lane == 0) sm.count[warp] = rows;
      __syncthreads();
      rows = 0;
#pragma unroll
      for (int w = 0; w < kTileWarps; w++) rows += sm.count[w];
    }
    const int n_cta = sm.n_cta, n_warp = sm.n_warp;

    for (int panel = blockIdx.y; panel < t.panels; panel += gridDim.y) {
    const int col0 = panel * (L * W * VEC) + l * W;
    bool col_ok[VEC];
    const char* Bcol[VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) {
      col_ok[v] = (col0 + v * L * W) < a.k;
      Bcol[v] = reinterpret_cast<const char*>(a.B + (col_ok[v] ? col0 + v * L * W : 0));
    }

    for (int i = 0; i < n_cta; i++) {
      const TileUnit q = sm.by_cta[i];
      const int slice = (q.len + NG - 1) / NG, w0 = min(q.len, (warp * G + g) * slice);
      const int b = q.begin - e0 + w0;
      Pack<T, W> s[VEC];
      // (a row of several units gets its present contents from the kernel that adds the units)
      tile_begin_row<T, L, VEC, W>(s, a, q.row, col0, col_ok, warp == 0 && lane < L && q.whole);
      tile_add<T, VEC, W, U>(s, sm.entry, b, b + min(slice, q.len - w0), Bcol, pitch);
      reduce_groups<T, L, VEC, W>(s);
      if (lane < L) {
#pragma unroll
        for (int v = 0; v < VEC; v++) sm.part[warp][v][l] = s[v];
      }
      __syncthreads();
      if (warp == (i % kTileWarps) && lane < L) {
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          s[v] = sm.part[0][v][l];
#pragma unroll
          for (int w2 = 1; w2 < kTileWarps; w2++) {
            const Pack<T, W> x = sm.part[w2][v][l];
#pragma unroll
            for (int w = 0; w < W; w++) s[v].v[w] += x.v[w];
          }
        }
        if (q.whole) {
          tile_store_row<T, L, VEC, W>(a, q.row, col0, col_ok, s);
        } else {
          T* dst = (q.begin == __ldg(a.pos + q.row) ? t.first : t.rest) + (long long)(q.begin / kUnit) * a.k + col0;
#pragma unroll
          for (int v = 0; v < VEC; v++)
            if (col_ok[v]) store_plain<T, W>(dst + v * L * W, s[v]);
        }
      }
      __syncthreads();
    }

    while (true) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&sm.next_warp, 1);
      i = __shfl_sync(FULL, i, 0);
      if (i >= n_warp) break;
      const TileUnit q = sm.by_warp[i];
      const int slice = (q.len + G - 1) / G, w0 = min(q.len, g * slice);
      const int b = q.begin - e0 + w0;
      Pack<T, W> s[VEC];
      tile_begin_row<T, L, VEC, W>(s, a, q.row, col0, col_ok, lane < L);
      tile_add<T, VEC, W, U>(s, sm.entry, b, b + min(slice, q.len - w0), Bcol, pitch);
      reduce_groups<T, L, VEC, W>(s);
      if (lane < L) tile_store_row<T, L, VEC, W>(a, q.row, col0, col_ok, s);
    }

    while (true) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&sm.next_row, G);
      i = __shfl_sync(FULL, i, 0);
      if (i >= rows) break;
      i += g;
      if constexpr (G > 1) {
        if (i >= rows) continue;
        int c = 0, before = 0;
#pragma unroll
        for (int q = 0; q + 1 < kShortClasses; q++) {
          c += i >= n_short[q];
          before = i >= n_short[q] ? n_short[q] : before;
        }
        i = sm.short_row[c >> 1][c & 1 ? kTileRowCap - 1 - (i - before) : i - before];
      }
      const int b = sm.pos[i], len = sm.pos[i + 1] - b;
      if (G == 1 && (b < next || len == 0 || len > kGroupRow<L>)) continue;
      Pack<T, W> s[VEC];
      tile_begin_row<T, L, VEC, W>(s, a, r0 + i, col0, col_ok, true);
      tile_add<T, VEC, W, U>(s, sm.entry, b - e0, b - e0 + len, Bcol, pitch);
      tile_store_row<T, L, VEC, W>(a, r0 + i, col0, col_ok, s);
    }
    __syncthreads();
    if (tid == 0) sm.next_warp = sm.next_row = 0;
    __syncthreads();
    }
    next = sm.pos[kTileRowCap];
    __syncthreads();
  }
}

// Rows without entries (zeros, or act(bias)), and rows of several units: their unit sums, every eighth one added in
// order, then these eight sums.  A warp looks at 32 rows and takes those that need something, a lane per column.
// Rows of more than kCtaUnits units are taken by the CTA, a warp per eighth: by one warp the rows of 90,000
// entries of a power-law matrix kept the product waiting (150,000 rows, 128 columns: 186 us, 172 so; one row of
// 130,000, 8 columns: 50.9 us, 10.6).  Shorter ones stay with the warps, which take eight rows at a time (200 rows
// of 5,000 entries, 8 columns, us: 170.9 with 8 units as the limit, 38.5 with 16; 30 of 4,200: 30.1, 26.6; 30 of
// 9,000: 38.4 both).  Small products take this form too: one without the CTA's part, whose row pointers were
// waited for behind the tile kernel, took longer (2,500 rows of 5 entries, 8 columns: 5.0 us, 4.5 this way).
constexpr int kWarpUnits = 8, kCtaUnits = 16;
static_assert(kWarpUnits == kTileWarps, "a warp per part");
template <typename T>
__global__ void __launch_bounds__(kTileThreadsMm)
spmm_tile_rows_kernel(SpmmArgs<T> a, TileArgs<T> t) {
  __shared__ int s_rows[kTileThreadsMm], s_n;
  __shared__ T s_part[kTileWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (what follows waits for this kernel's end)
  const long long r0 = ((long long)blockIdx.x * kTileWarps + warp) * 32;
  int b = 0, len = 1;
  if (r0 + lane < a.m) {
    b = __ldg(a.pos + r0 + lane);
    len = __ldg(a.pos + r0 + lane + 1) - b;
  }
  // (an empty row of an accumulating product without bias or ReLU stays what it is)
  const bool keep_empty = a.accumulate && !a.bias && !a.relu, by_cta = len > kCtaUnits * kUnit;
  unsigned todo = __ballot_sync(FULL, (len == 0 && !keep_empty) || (len > kUnit && !by_cta));
  if (threadIdx.x == 0) s_n = 0;
  const bool some = __syncthreads_or(by_cta);
  if (by_cta) s_rows[atomicAdd(&s_n, 1)] = (int)(r0 + lane);
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the tile kernel's results
  auto unit_sum = [&](int rb, int u, int col) {
    return (u ? t.rest : t.first)[((long long)(rb / kUnit) + u) * a.k + col];
  };
  auto store = [&](T* c, int col, T s) {
    Pack<T, 1> x;
    x.v[0] = s + (a.accumulate ? *c : T(0));
    st_stream<T, 1>(c, epilogue<T, 1>(x, a.bias, col, a.relu));
  };
  while (todo) {
    const int i = __ffs(todo) - 1;
    todo &= todo - 1;
    const int rb = __shfl_sync(FULL, b, i), units = (__shfl_sync(FULL, len, i) + kUnit - 1) / kUnit;
    T* crow = a.C + (r0 + i) * a.ldc;
    for (int col = blockIdx.y * 32 + lane; col < a.k; col += gridDim.y * 32) {
      T s[kWarpUnits];
#pragma unroll
      for (int w = 0; w < kWarpUnits; w++) s[w] = w < units ? unit_sum(rb, w, col) : T(0);
      for (int u = kWarpUnits; u < units; u += kWarpUnits) {
#pragma unroll
        for (int w = 0; w < kWarpUnits; w++)
          if (u + w < units) s[w] += unit_sum(rb, u + w, col);
      }
      T sum = s[0];
#pragma unroll
      for (int w = 1; w < kWarpUnits; w++)
        if (w < units) sum += s[w];
      store(crow + col, col, sum);
    }
  }
  if (!some) return;
  __syncthreads();
  for (int i = 0; i < s_n; i++) {
    const int r = s_rows[i], rb = __ldg(a.pos + r), units = (__ldg(a.pos + r + 1) - rb + kUnit - 1) / kUnit;
    for (int col0 = blockIdx.y * 32; col0 < a.k; col0 += gridDim.y * 32) {
      const int col = col0 + lane;
      if (col < a.k) {
        T s = unit_sum(rb, warp, col);
#pragma unroll 8
        for (int u = warp + kWarpUnits; u < units; u += kWarpUnits) s += unit_sum(rb, u, col);
        s_part[warp][lane] = s;
      }
      __syncthreads();
      if (warp == 0 && col < a.k) {
        T s = s_part[0][lane];
#pragma unroll
        for (int w = 1; w < kTileWarps; w++) s += s_part[w][lane];
        store(a.C + (long long)r * a.ldc + col, col, s);
      }
      __syncthreads();
    }
  }
}

// (two unit sums per kUnit entries)
inline size_t tile_workspace_bytes(size_t size, int64_t k, int64_t nnz) {
  return nnz <= kUnit ? 0 : 2 * (size_t)(nnz / kUnit + 1) * (size_t)k * size;
}

template <typename T, int L, int VEC, int W>
static int launch_tiles(const SpmmArgs<T>& a, int64_t nnz, void* ws, cudaStream_t st) {
  using Smem = TileSmem<T, L, VEC, W>;
  const unsigned panels = (unsigned)ceil_div(a.k, L * W * VEC);
  if (panels > 65535)
    return fail(SB_ERR_UNSUPPORTED, "spmm: at most %lld columns with this layout, got %d",
                65535ll * (L * W * VEC), a.k);
  TileArgs<T> t;
  t.nnz = (int)nnz;
  t.panels = (int)panels;
  // Column panels.  An operand that L2 holds whole: every (window, panel) is a CTA of its own, windows
  // sized for all of them together (81,724 entries, 8 panels of 4 MB: 63 us with the next form, 45
  // with this).  A larger one, all windows resident at once: every CTA goes through the panels
  // itself; its start-up is paid once, and the CTAs, equally loaded, stay at about the same panel,
  // which L2 holds (262,144 entries, 16 panels of 32 MB: 286 us panel by panel, 249 this way).
  // Otherwise panel after panel on grid.y.
  const bool in_l2 = (double)a.n * a.ldb * sizeof(T) <= 64e6;
  t.entries = tile_entries(in_l2 ? nnz * panels : nnz, L, sizeof(T));
  t.tiles = (int)ceil_div(nnz, t.entries);
  t.first = static_cast<T*>(ws);
  t.rest = t.first + (size_t)(nnz / kUnit + 1) * a.k;
  if (t.tiles > 0) {
    auto kernel = spmm_tile_kernel<T, L, VEC, W>;
    static bool sized[64] = {};   // per device: the attribute is set once
    int dev = 0;
    SB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !sized[dev]) {
      SB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
      if (dev >= 0 && dev < 64) sized[dev] = true;
    }
    const bool resident = !in_l2 && t.tiles <= sm_count() * tile_ctas(L);
    SB_CUDA(launch_early(kernel, dim3((unsigned)t.tiles, resident ? 1 : panels), kTileThreadsMm, sizeof(Smem), st, a, t));
  }
  // (may be set up while the tiles still run: it waits for them itself.  It reads the row pointers before
  // that, which is sound behind the tile kernel, whose CTAs have waited for whatever made them; a
  // matrix without entries has no tile kernel, and an ordinary launch)
  const dim3 grid((unsigned)ceil_div(a.m, kTileThreadsMm), (unsigned)std::min<int64_t>(ceil_div(a.k, 32), 64));
  SB_CUDA(launch_kernel(t.tiles > 0, spmm_tile_rows_kernel<T>, grid, kTileThreadsMm, 0, st, a, t));
  return SB_OK;
}

}  // namespace sb
