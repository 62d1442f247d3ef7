// Column split of a CSR matrix: chunk c holds the entries whose columns lie in [c * width, (c + 1) * width),
// as a CSR matrix of the same rows.  A product with a dense operand far larger than L2 then runs
// chunk after chunk over operand rows that stay in L2 (accumulating into the result) instead of
// gathering every entry's row from DRAM.  Column indices are kept, so every chunk multiplies the
// same operand.
//
// Columns ascend within a row, so a row's entries of a chunk are consecutive: their bounds are binary
// searches, the new row pointers one scan over chunk-major counts, and the entries move in one pass
// balanced by entries.  The pass checks that the columns ascend; a matrix where they do not is
// reported and not split.
// Bound: DRAM, 16 bytes per entry moved and 4 searched (2 M rows, 202 M entries: 1.2 ms).
#include <algorithm>

#include "common.cuh"

namespace sb {

constexpr int kMaxChunks = 64;
// Entries and row pointers that a CTA of the move has at a time; entries per thread whose loads are in flight together.
constexpr int kTile = 8192, kTileRows = 1024, kAhead = 4;

// Bounds and counts of row r: first[c * m + r] = its first entry of chunk c.
__global__ void __launch_bounds__(256)
split_bounds_kernel(int m, int chunks, int width, const int* __restrict__ pos, const int* __restrict__ crd,
                    int* __restrict__ first, int* __restrict__ cnt) {
  const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
  if (r >= m) return;
  const int e = __ldg(pos + r + 1);
  int at = __ldg(pos + r);
  for (int c = 0; c < chunks; c++) {
    int lo = at, hi = e;
    if (c + 1 < chunks) {
      const int limit = (c + 1) * width;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(crd + mid) < limit) lo = mid + 1; else hi = mid;
      }
    } else {
      lo = e;
    }
    first[(long long)c * m + r] = at;
    cnt[(long long)c * m + r] = lo - at;
    at = lo;
  }
}

// Row pointers per chunk, counted from the chunk's own start; first[] becomes the way of the row's
// entries of a chunk: new place - old place.
__global__ void __launch_bounds__(256)
split_pos_kernel(int m, int chunks, const int* __restrict__ flat, int* __restrict__ rpos, int* __restrict__ first,
                 int* __restrict__ ends) {
  const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
  if (r > m) return;
  for (int c = 0; c < chunks; c++) {
    const int at = __ldg(flat + (long long)c * m + r);
    rpos[(long long)c * (m + 1) + r] = at - __ldg(flat + (long long)c * m);
    if (r == m) ends[c] = at - __ldg(flat + (long long)c * m);
    if (r < m) first[(long long)c * m + r] = at - first[(long long)c * m + r];
  }
}

// A CTA moves kTile consecutive entries; the rows of kAhead times 32 of them are looked up in shared memory, then all
// of them are loaded, then stored.  (A warp that walked along its entries' rows, 32 entries at a time, had 256 bytes
// in flight: 1.26 ms for 202 M entries, 0.89 so.)
__global__ void __launch_bounds__(256)
split_move_kernel(int m, int nnz, int chunks, int width, const int* __restrict__ pos, const int* __restrict__ crd,
                  const float* __restrict__ val, const int* __restrict__ way, int* __restrict__ ccrd,
                  float* __restrict__ cval, int* __restrict__ unsorted) {
  __shared__ int s_pos[kTileRows + 1], s_first[kTileRows / 32], s_count[8];
  const int tid = threadIdx.x, lane = tid & 31;
  const int e1 = (int)min((long long)nnz, ((long long)blockIdx.x + 1) * kTile);
  const float inv = 1.f / (float)width;
  bool bad = false;
  for (int e = blockIdx.x * kTile; e < e1;) {
    const int r0 = cta_row_of<256>(pos, m, e, s_count);
    for (int x = tid; x < kTileRows + 1; x += 256) {
      const int p = __ldg(pos + min(m, r0 + x));
      s_pos[x] = p;
      if (x % 32 == 0 && x < kTileRows) s_first[x / 32] = p;
    }
    __syncthreads();
    const int stop = min(e1, s_pos[kTileRows]);
    for (int o0 = e + (tid & ~31); o0 < stop; o0 += 256 * kAhead) {
      int row[kAhead], col[kAhead], left[kAhead];
      float v[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; q++) {
        const int o = o0 + q * 256 + lane;
        col[q] = left[q] = 0;
        v[q] = 0.f;
        if (o < stop) {
          col[q] = ld_stream(crd + o);
          v[q] = ld_stream(val + o);
          if (lane == 0 && o > 0) left[q] = __ldg(crd + o - 1);
        }
      }
#pragma unroll
      for (int q = 0; q < kAhead; q++) {
        // the row of the warp's first entry by two rounds of 32 looks, this lane's a few rows behind it
        const int first = min(o0 + q * 256, stop - 1), o = min(first + lane, stop - 1);
        const int c = __popc(__ballot_sync(FULL, s_first[lane] <= first)) - 1;
        int r = 32 * c + __popc(__ballot_sync(FULL, s_pos[32 * c + lane] <= first)) - 1;
#pragma unroll 1
        for (int step = 0; step < 6 && s_pos[r + 1] <= o; step++) r++;
        if (s_pos[r + 1] <= o) {           // many short or empty rows
          int hi = kTileRows;
          while (hi - r > 1) {
            const int mid = (r + hi) >> 1;
            if (s_pos[mid] <= o) r = mid; else hi = mid;
          }
        }
        row[q] = r;
        const int before = __shfl_up_sync(FULL, col[q], 1);
        if (lane > 0) left[q] = before;
      }
      int dst[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; q++) {
        const int o = o0 + q * 256 + lane;
        dst[q] = -1;
        if (o >= stop) continue;
        if (s_pos[row[q]] < o && left[q] > col[q]) bad = true;
        int c = (int)((float)col[q] * inv);                 // col / width, one off at most
        c += (c + 1ll) * width <= col[q];
        c -= (long long)c * width > col[q];
        dst[q] = o + __ldg(way + (long long)c * m + r0 + row[q]);
      }
#pragma unroll
      for (int q = 0; q < kAhead; q++) {
        if ((unsigned)dst[q] < (unsigned)nnz) {             // (always, where the columns ascend)
          ccrd[dst[q]] = col[q];
          cval[dst[q]] = v[q];
        }
      }
    }
    e = stop;
    __syncthreads();
  }
  if (__any_sync(FULL, bad) && lane == 0) *unsorted = 1;
}

struct SplitWs {
  int *first, *cnt, *flat;
  long long *block_sum, *total;
  int *unsorted, *ends;   // (neighbours: one copy to the host)
  size_t bytes;
};
static SplitWs split_ws(void* base, int64_t m, int64_t chunks) {
  SplitWs w;
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t b) { char* q = p + off; off += (b + 255) / 256 * 256; return q; };
  const size_t cells = (size_t)m * (size_t)chunks;
  w.first = (int*)take(cells * 4);
  w.cnt = (int*)take(cells * 4);
  w.flat = (int*)take((cells + 1) * 4);
  w.block_sum = (long long*)take((size_t)(ceil_div((int64_t)cells, 4096) + 1) * 8);
  w.total = (long long*)take(8);
  w.unsorted = (int*)take((1 + kMaxChunks) * 4);
  w.ends = w.unsorted + 1;
  w.bytes = off;
  return w;
}

}  // namespace sb

using namespace sb;

extern "C" {

size_t sb_csr_split_columns_workspace_bytes(int64_t m, int64_t chunks) {
  return split_ws(nullptr, m < 0 ? 0 : m, chunks < 1 ? 1 : chunks).bytes;
}

int sb_csr_split_columns_f32(int64_t m, int64_t n, int64_t nnz, const int32_t* pos, const int32_t* crd,
                             const float* val, int64_t chunks, int32_t* rpos, int32_t* ccrd, float* cval,
                             int64_t* counts_host, void* ws, size_t ws_bytes, void* stream) {
  SB_CHECK_ARG(m > 0 && n > 0 && nnz > 0 && m < INT32_MAX && n < INT32_MAX, "csr_split: bad size");
  SB_CHECK_ARG(chunks >= 1 && chunks <= kMaxChunks && m * chunks < INT32_MAX - 4096, "csr_split: too many chunks");
  if (nnz > INT32_MAX - 4096) return fail(SB_ERR_OVERFLOW, "csr_split: nnz=%lld does not fit int32", (long long)nnz);
  SB_CHECK_ARG(pos && crd && val && rpos && ccrd && cval && counts_host, "csr_split: null pointer");
  SB_CHECK_ARG(ws && aligned16(ws), "csr_split: workspace is null or misaligned");
  const SplitWs w = split_ws(ws, m, chunks);
  if (ws_bytes < w.bytes)
    return fail(SB_ERR_WORKSPACE, "csr_split: workspace has %zu bytes, needs %zu", ws_bytes, w.bytes);
  cudaStream_t st = (cudaStream_t)stream;
  const int width = (int)ceil_div(n, chunks);
  SB_CUDA(cudaMemsetAsync(w.unsorted, 0, 4, st));
  split_bounds_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>((int)m, (int)chunks, width, pos, crd, w.first, w.cnt);
  SB_LAUNCH_CHECK("split_bounds_kernel");
  int rc = exclusive_scan_i32((int)(m * chunks), w.cnt, w.flat, w.block_sum, w.total, st);
  if (rc != SB_OK) return rc;
  split_pos_kernel<<<(unsigned)ceil_div(m + 1, 256), 256, 0, st>>>((int)m, (int)chunks, w.flat, rpos, w.first, w.ends);
  SB_LAUNCH_CHECK("split_pos_kernel");
  split_move_kernel<<<(unsigned)ceil_div(nnz, kTile), 256, 0, st>>>((int)m, (int)nnz, (int)chunks, width, pos, crd,
                                                                        val, w.first, ccrd, cval, w.unsorted);
  SB_LAUNCH_CHECK("split_move_kernel");
  int host[1 + kMaxChunks];
  SB_CUDA(cudaMemcpyAsync(host, w.unsorted, (size_t)(1 + chunks) * 4, cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  if (host[0]) return fail(SB_ERR_UNSUPPORTED, "csr_split: the columns of a row do not ascend");
  for (int c = 0; c < chunks; c++) counts_host[c] = host[1 + c];
  return SB_OK;
}

}  // extern "C"
