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
// Bound: DRAM, 16 bytes per entry moved and 4 searched (2 M rows, 202 M entries: 1.3 ms).
#include <algorithm>

#include "common.cuh"

namespace sb {

constexpr int kMaxChunks = 64;
constexpr int kSpan = 1024;      // consecutive entries per warp

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
split_pos_kernel(int m, int chunks, const int* __restrict__ flat, int* __restrict__ rpos, int* __restrict__ first) {
  const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
  if (r > m) return;
  for (int c = 0; c < chunks; c++) {
    const int at = __ldg(flat + (long long)c * m + r);
    rpos[(long long)c * (m + 1) + r] = at - __ldg(flat + (long long)c * m);
    if (r < m) first[(long long)c * m + r] = at - first[(long long)c * m + r];
  }
}

__global__ void __launch_bounds__(256)
split_move_kernel(int m, int nnz, int chunks, int width, const int* __restrict__ pos, const int* __restrict__ crd,
                  const float* __restrict__ val, const int* __restrict__ way, int* __restrict__ ccrd,
                  float* __restrict__ cval, int* __restrict__ unsorted) {
  const int lane = threadIdx.x & 31;
  const long long p_begin = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * kSpan;
  if (p_begin >= nnz) return;
  const int p_end = (int)min((long long)nnz, p_begin + kSpan);
  // the span's first row, the warp together
  int lo = 0, hi = m;
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32;
    const long long r = (long long)lo + (long long)lane * step;
    const unsigned le = __ballot_sync(FULL, r < hi && __ldg(pos + r) <= (int)p_begin);
    lo += (__popc(le) - 1) * step;
    hi = min(hi, lo + step);
  }
  int r0 = lo;
  bool bad = false;
  int last_col = -1, last_row = -1;    // of the entry before the group
  if (p_begin > 0) {
    last_col = __ldg(crd + p_begin - 1);
    last_row = __ldg(pos + r0) <= (int)p_begin - 1 ? r0 : -1;
  }
  const float inv = 1.f / (float)width;
  for (int p0 = (int)p_begin; p0 < p_end; p0 += 32) {
    const int p = p0 + lane;
    const bool in = p < p_end;
    int col = 0;
    float v = 0.f;
    if (in) {
      col = ld_stream(crd + p);
      v = ld_stream(val + p);
    }
    // the row of this lane's entry: forward from the row of the group's first one
    int r = r0;
    while (in && __ldg(pos + r + 1) <= p) r++;
    int before_col = __shfl_up_sync(FULL, col, 1), before_row = __shfl_up_sync(FULL, r, 1);
    if (lane == 0) { before_col = last_col; before_row = last_row; }
    if (in) {
      if (before_row == r && before_col > col) bad = true;
      int c = (int)((float)col * inv);                    // col / width, one off at most
      c += (c + 1ll) * width <= col;
      c -= (long long)c * width > col;
      const int dst = p + __ldg(way + (long long)c * m + r);
      if ((unsigned)dst < (unsigned)nnz) {                // (always, where the columns ascend)
        ccrd[dst] = col;
        cval[dst] = v;
      }
    }
    const int n = min(31, p_end - 1 - p0);
    r0 = last_row = __shfl_sync(FULL, r, n);
    last_col = __shfl_sync(FULL, col, n);
  }
  if (__any_sync(FULL, bad) && lane == 0) *unsorted = 1;
}

struct SplitWs {
  int *first, *cnt, *flat;
  long long *block_sum, *total;
  int* unsorted;
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
  w.unsorted = (int*)take(4);
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
  split_pos_kernel<<<(unsigned)ceil_div(m + 1, 256), 256, 0, st>>>((int)m, (int)chunks, w.flat, rpos, w.first);
  SB_LAUNCH_CHECK("split_pos_kernel");
  split_move_kernel<<<(unsigned)ceil_div(nnz, 8 * kSpan), 256, 0, st>>>((int)m, (int)nnz, (int)chunks, width, pos, crd,
                                                                        val, w.first, ccrd, cval, w.unsorted);
  SB_LAUNCH_CHECK("split_move_kernel");
  int ends[kMaxChunks], unsorted = 0;
  for (int c = 0; c < chunks; c++)
    SB_CUDA(cudaMemcpyAsync(&ends[c], rpos + (int64_t)c * (m + 1) + m, 4, cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaMemcpyAsync(&unsorted, w.unsorted, 4, cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  if (unsorted) return fail(SB_ERR_UNSUPPORTED, "csr_split: the columns of a row do not ascend");
  for (int c = 0; c < chunks; c++) counts_host[c] = ends[c];
  return SB_OK;
}

}  // extern "C"
