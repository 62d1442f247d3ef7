// CSR SpMV for sm_100a.
//
// Entry-tiled kernel (below), balanced by stored entries.  x is gathered through the
// read-only path (it is L2 resident: 8 MB for 2M columns); the CSR streams are read once with
// no-allocate loads.  The entry point without scratch (sb_spmv_csr_typed) uses a plain
// G-lanes-per-row kernel (G chosen from the mean row length).
#include "common.cuh"

namespace sb {

template <typename T>
__device__ __forceinline__ T shfl_xor_t(T v, int o) { return __shfl_xor_sync(FULL, v, o); }

template <typename T, int G>
__global__ void __launch_bounds__(256)
spmv_rows_kernel(int m, const int* __restrict__ pos, const int* __restrict__ crd,
                 const T* __restrict__ val, const T* __restrict__ x, T* __restrict__ y) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = t / G;
  const int l = (int)(t % G);
  T acc = T(0);
  if (row < m) {
    const int b = __ldg(pos + row), e = __ldg(pos + row + 1);
    for (int p = b + l; p < e; p += G) acc += val[p] * __ldg(x + crd[p]);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) acc += shfl_xor_t(acc, o);
  if (row < m && l == 0) y[row] = acc;
}

// ---- entry-tiled kernel --------------------------------------------------------------------------
// The entry arrays are cut into tiles of kTile consecutive entries, one CTA per tile, whatever
// the row lengths are (power-law rows included: a hub row simply spans many tiles).  A first, small
// kernel notes the row of every tile's first entry.  A tile
//   1. streams its crd/val slices with 8 independent loads per thread, gathers x and leaves the
//      products in shared memory,
//   2. sums each row's segment (one thread per row for short rows, one warp per row for long
//      ones) and writes y for rows that lie completely inside the tile, empty ones included.
// A row cut by a tile border leaves partial sums in the scratch arrays; a third kernel adds them in
// tile order, so the result does not depend on scheduling.
// Bound: the gather of x, one L1 tag look-up per entry and clock and SM (288 G entries/s measured for
// random 4-byte loads: 83 us for the 23.8 M entries of a 2 M-row power-law matrix).  A search for the
// rows in every tile, 256 scattered loads a round, took nearly as many look-ups as the gather: 174 us;
// 129 us with the rows noted beforehand.
constexpr int kTile = 2048;
constexpr int kTileThreads = 256;

template <typename T>
struct TileScratch {
  T* carry_first;   // partial sum of the tile's first row when that row began in an earlier tile
  T* carry_last;    // partial sum of the tile's last row when it began here and continues
  int* row;         // row of the tile's first entry (0 for the first tile)
};

// (rows that end behind a tile's start and begin at or before it)
__global__ void __launch_bounds__(256)
spmv_tile_rows_kernel(int m, int tiles, const int* __restrict__ pos, int* __restrict__ row) {
  const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the tiles' products do not need this kernel
  if (r >= m) return;
  const int b = __ldg(pos + r), e = __ldg(pos + r + 1);
  if (r == 0) row[0] = 0;
  for (int t = (b + kTile - 1) / kTile; t < tiles && (long long)t * kTile < e; t++)
    if (t > 0) row[t] = (int)r;
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
__global__ void __launch_bounds__(kTileThreads)
spmv_tile_kernel(int m, int nnz, int tiles, const int* __restrict__ pos, const int* __restrict__ crd,
                 const T* __restrict__ val, const T* __restrict__ x, T* __restrict__ y, TileScratch<T> sc) {
  __shared__ T prod[kTile];
  const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int e0 = t * kTile, e1 = min(nnz, e0 + kTile);
  // products first: they do not need the rows
  {
    int j[kTile / kTileThreads];
    T a[kTile / kTileThreads];
#pragma unroll
    for (int q = 0; q < kTile / kTileThreads; q++) {
      const int e = e0 + tid + q * kTileThreads;
      j[q] = 0;
      a[q] = T(0);
      if (e < e1) {
        j[q] = ld_stream(crd + e);
        a[q] = ld_stream(val + e);
      }
    }
#pragma unroll
    for (int q = 0; q < kTile / kTileThreads; q++) {
      const int e = e0 + tid + q * kTileThreads;
      prod[tid + q * kTileThreads] = (e < e1) ? a[q] * __ldg(x + j[q]) : T(0);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the tiles' rows
  const int r_lo = sc.row[t], r_hi = t + 1 < tiles ? sc.row[t + 1] : m - 1;
  __syncthreads();
  const int nr = r_hi - r_lo + 1;
  const bool thread_per_row = nr >= 128;
  const int first = thread_per_row ? tid : warp;
  const int stride = thread_per_row ? kTileThreads : kTileThreads / 32;
  for (int r = r_lo + first; r <= r_hi; r += stride) {
    const int rb = __ldg(pos + r), re = __ldg(pos + r + 1);
    if (r == r_hi && rb >= e1 && t + 1 < tiles) continue;   // (begins with the next tile)
    const int b = max(rb, e0) - e0, e = min(re, e1) - e0;
    T s = T(0);
    if (thread_per_row) {
      for (int i = b; i < e; i++) s += prod[i];
    } else {
      for (int i = b + lane; i < e; i += 32) s += prod[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
      if (lane != 0) continue;
    }
    if (rb >= e0 && re <= e1) {
      y[r] = s;
    } else if (rb < e0) {
      sc.carry_first[t] = s;             // continues a row that began in an earlier tile
    } else {
      sc.carry_last[t] = s;              // begins here, continues in the next tile
    }
  }
}

// Adds the pieces of every row that was cut by tile borders, in tile order.
template <typename T>
__global__ void spmv_tile_fixup_kernel(int ntiles, const int* __restrict__ pos, T* __restrict__ y, TileScratch<T> sc) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (t + 1 >= ntiles) return;
  // the row that the next tile begins with, if it began in this tile
  const int r = sc.row[t + 1];
  const int rb = __ldg(pos + r), re = __ldg(pos + r + 1);
  if (rb >= (t + 1) * kTile || rb < t * kTile) return;
  T s = sc.carry_last[t];
  const int last = (re - 1) / kTile;
#pragma unroll 8
  for (int u = t + 1; u <= last; u++) s += sc.carry_first[u];
  y[r] = s;
}

template <typename T>
static int launch_tiles(int64_t m, int64_t nnz, const int32_t* pos, const int32_t* crd, const T* val, const T* x,
                        T* y, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  const int tiles = (int)ceil_div(nnz, kTile);
  const size_t stride = scratch_bytes / 3 / 256 * 256;
  char* base = static_cast<char*>(scratch);
  TileScratch<T> sc{reinterpret_cast<T*>(base), reinterpret_cast<T*>(base + stride),
                    reinterpret_cast<int*>(base + 2 * stride)};
  spmv_tile_rows_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>((int)m, tiles, pos, sc.row);
  SB_LAUNCH_CHECK("spmv_tile_rows_kernel");
  SB_CUDA(launch_early(spmv_tile_kernel<T>, dim3((unsigned)tiles), kTileThreads, 0, st, (int)m, (int)nnz, tiles, pos,
                       crd, val, x, y, sc));
  if (tiles > 1)
    SB_CUDA(launch_early(spmv_tile_fixup_kernel<T>, dim3((unsigned)ceil_div(tiles, 128)), 128, 0, st, tiles, pos, y, sc));
  return SB_OK;
}

template <typename T>
static int launch_rows(int64_t m, int64_t nnz, const int32_t* pos, const int32_t* crd,
                       const T* val, const T* x, T* y, cudaStream_t st) {
  const double mean = m > 0 ? (double)nnz / (double)m : 0.0;
  const int threads = 256;
#define SB_SPMV_LAUNCH(G)                                                                    \
  spmv_rows_kernel<T, G><<<(unsigned)ceil_div(m * (int64_t)G, threads), threads, 0, st>>>(   \
      (int)m, pos, crd, val, x, y)
  if (mean <= 3.0) SB_SPMV_LAUNCH(2);
  else if (mean <= 6.0) SB_SPMV_LAUNCH(4);
  else if (mean <= 12.0) SB_SPMV_LAUNCH(8);
  else if (mean <= 48.0) SB_SPMV_LAUNCH(16);
  else SB_SPMV_LAUNCH(32);
#undef SB_SPMV_LAUNCH
  SB_LAUNCH_CHECK("spmv_rows_kernel");
  return SB_OK;
}

static int check_spmv(int64_t m, int64_t n, int64_t nnz, const void* pos, const void* crd,
                      const void* val, const void* x, const void* y) {
  SB_CHECK_ARG(m >= 0 && n >= 0 && nnz >= 0, "spmv: negative size");
  SB_CHECK_ARG(m < INT32_MAX / 32 * 32 && n < INT32_MAX, "spmv: dimension exceeds int32");
  // (the tile kernels add up to one tile, 2048 entries, to an entry index held in an int)
  if (nnz > INT32_MAX - 4096)
    return fail(SB_ERR_OVERFLOW, "spmv: nnz=%lld does not fit int32 row pointers", (long long)nnz);
  SB_CHECK_ARG(pos, "spmv: pos is null");
  SB_CHECK_ARG(nnz == 0 || (crd && val && x), "spmv: null crd/val/x");
  SB_CHECK_ARG(m == 0 || y, "spmv: y is null");
  return SB_OK;
}

}  // namespace sb

using namespace sb;

extern "C" {

size_t sb_spmv_csr_scratch_bytes(int64_t nnz) {
  if (nnz <= 0) return 0;
  const size_t tiles = (size_t)ceil_div(nnz, kTile);
  return ((tiles * 4 + 255) / 256 * 256) * 3;
}

size_t sb_spmv_csr_tiled_scratch_bytes(int dtype, int64_t nnz) {
  if (nnz <= 0) return 0;
  const size_t tiles = (size_t)ceil_div(nnz, kTile);
  return ((tiles * (dtype == SB_F64 || dtype == SB_I64 ? 8 : 4) + 255) / 256 * 256) * 3;
}

int sb_spmv_csr_tiled(int dtype, int64_t m, int64_t n, int64_t nnz, const int32_t* pos, const int32_t* crd,
                      const void* val, const void* x, void* y, void* scratch, size_t scratch_bytes, void* stream) {
  int rc = check_spmv(m, n, nnz, pos, crd, val, x, y);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(dtype >= SB_F32 && dtype <= SB_I64, "spmv: unknown dtype %d", dtype);
  if (m == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool wide = dtype == SB_F64 || dtype == SB_I64;
  if (nnz == 0) {
    SB_CUDA(cudaMemsetAsync(y, 0, (size_t)m * (wide ? 8 : 4), st));
    return SB_OK;
  }
  const size_t need = sb_spmv_csr_tiled_scratch_bytes(dtype, nnz);
  SB_CHECK_ARG(scratch && aligned16(scratch), "spmv: scratch is null or misaligned");
  if (scratch_bytes < need)
    return fail(SB_ERR_WORKSPACE, "spmv: scratch has %zu bytes, needs %zu", scratch_bytes, need);
  switch (dtype) {
    case SB_F32:
      return launch_tiles<float>(m, nnz, pos, crd, (const float*)val, (const float*)x, (float*)y, scratch, need, st);
    case SB_F64:
      return launch_tiles<double>(m, nnz, pos, crd, (const double*)val, (const double*)x, (double*)y, scratch, need, st);
    case SB_I32:  // unsigned arithmetic: same bits as the reference's wrapping int32 math
      return launch_tiles<unsigned int>(m, nnz, pos, crd, (const unsigned int*)val, (const unsigned int*)x,
                                        (unsigned int*)y, scratch, need, st);
    default:
      return launch_tiles<unsigned long long>(m, nnz, pos, crd, (const unsigned long long*)val,
                                              (const unsigned long long*)x, (unsigned long long*)y, scratch, need, st);
  }
}

int sb_spmv_csr_f32(int64_t m, int64_t n, int64_t nnz, const int32_t* pos, const int32_t* crd,
                    const float* val, const float* x, float* y, void* scratch, size_t scratch_bytes,
                    void* stream) {
  return sb_spmv_csr_tiled(SB_F32, m, n, nnz, pos, crd, val, x, y, scratch, scratch_bytes, stream);
}

int sb_spmv_csr_typed(int dtype, int64_t m, int64_t n, int64_t nnz, const int32_t* pos,
                      const int32_t* crd, const void* val, const void* x, void* y, void* stream) {
  int rc = check_spmv(m, n, nnz, pos, crd, val, x, y);
  if (rc != SB_OK) return rc;
  if (m == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  switch (dtype) {
    case SB_F32:  // without scratch: the lanes-per-row kernel
      return launch_rows<float>(m, nnz, pos, crd, (const float*)val, (const float*)x, (float*)y, st);
    case SB_F64:
      return launch_rows<double>(m, nnz, pos, crd, (const double*)val, (const double*)x, (double*)y, st);
    case SB_I32:  // unsigned arithmetic: same bits as the reference's wrapping int32 math
      return launch_rows<unsigned int>(m, nnz, pos, crd, (const unsigned int*)val,
                                       (const unsigned int*)x, (unsigned int*)y, st);
    case SB_I64:
      return launch_rows<unsigned long long>(m, nnz, pos, crd, (const unsigned long long*)val,
                                             (const unsigned long long*)x, (unsigned long long*)y, st);
    default:
      return fail(SB_ERR_UNSUPPORTED, "spmv_typed: unknown dtype %d", dtype);
  }
}

}  // extern "C"
