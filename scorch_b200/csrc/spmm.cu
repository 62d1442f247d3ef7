// CSR x dense SpMM for sm_100a: entry points and the fp32 forms with 16 and 32 byte loads (kernels
// in spmm_kernels.cuh).
#include "spmm_kernels.cuh"
#include "spmm_tiles.cuh"

namespace sb {

// Picks the kernel for the width and the widest load every row slice is aligned for: W elements
// per load, L lanes across a column tile, VEC loads per lane and entry; wider operands are cut
// into column panels on grid.y (256 columns: a 32768-row panel = 32 MB stays in L2 while all row
// blocks pass over it; 128- and 512-column panels measured slower).
int spmm_dispatch_f32(const SpmmArgs<float>& a, int64_t batch, const void* plan, int64_t nnz,
                      int64_t plan_segments, void* scratch, void* tile_ws, cudaStream_t st) {
  using T = float;
  const unsigned align = spmm_alignment(a);
  if (align < 16 || a.ldb >= (1ll << 32))
    return spmm_dispatch_f32_narrow(a, batch, plan, nnz, plan_segments, scratch, tile_ws, st);
  if (align == 32) {
    if (a.k <= 32) SB_GO_FIT(4, 1, 8);
    if (a.k <= 64) SB_GO_FIT(8, 1, 8);
    if (a.k <= 128) SB_GO_FIT(16, 1, 8);
    SB_GO_FIT(32, 1, 8);
  }
  if (a.k <= 16) SB_GO_FIT(4, 1, 4);
  if (a.k <= 32) SB_GO_FIT(8, 1, 4);
  if (a.k <= 64) SB_GO_FIT(16, 1, 4);
  if (a.k <= 128) SB_GO_FIT(32, 1, 4);
  SB_GO_FIT(32, 2, 4);
}

// Mean stored entries per row below which a launch takes several rows per warp.
static int short_rows_wanted(int64_t m, int64_t k, int64_t nnz) {
  return nnz < (int64_t)((k > 128 && k <= 256) ? SB_SPMM_SHORT_ROW_MEAN_FULL_WARP : SB_SPMM_SHORT_ROW_MEAN) * m;
}

template <typename T>
static SpmmArgs<T> spmm_args(int64_t m, int64_t n, int64_t k, int64_t nnz, const int* pos, const int* crd, const T* val,
                             const T* B, int64_t ldb, const T* bias, int relu, T* C, int64_t ldc,
                             int64_t stride_val, int64_t stride_b, int64_t stride_c) {
  SpmmArgs<T> a{};
  a.m = (int)m; a.n = (int)n; a.k = (int)k; a.pos = pos; a.end = pos + 1; a.crd = crd; a.val = val; a.B = B; a.ldb = ldb;
  a.bias = bias; a.relu = relu; a.C = C; a.ldc = ldc;
  a.stride_val = stride_val; a.stride_b = stride_b; a.stride_c = stride_c;
  a.short_rows = short_rows_wanted(m, k, nnz);
  return a;
}

// Rows of the entries outside the dense blocks of a block plan (blocked.cu): C += A_rem B, then
// bias / ReLU.  Entries are taken through the list `rem_ent`; no heavy-row split (the blocked
// path is only offered for matrices without heavy rows).
int spmm_remainder(int64_t m, int64_t k, const int* rem_pos, const int* rem_ent, const int* crd,
                   const float* val, const float* B, int64_t ldb, const float* bias, int relu,
                   float* C, int64_t ldc, int64_t batch, int64_t stride_val, int64_t stride_b,
                   int64_t stride_c, int val_compact, cudaStream_t st) {
  SpmmArgs<float> a = spmm_args<float>(m, m, k, 0, rem_pos, crd, val, B, ldb, bias, relu, C, ldc, stride_val,
                                       stride_b, stride_c);
  a.ent = rem_ent; a.val_compact = val_compact; a.accumulate = 1; a.short_rows = 1;
  return spmm_dispatch_f32(a, batch, nullptr, 0, 0, nullptr, nullptr, st);
}

static int check_common(int64_t m, int64_t n, int64_t k, int64_t nnz, const void* pos,
                        const void* crd, const void* val, const void* B, int64_t ldb,
                        const void* C, int64_t ldc) {
  SB_CHECK_ARG(m >= 0 && n >= 0 && k >= 0 && nnz >= 0, "spmm: negative size");
  SB_CHECK_ARG(m < INT32_MAX && n < INT32_MAX && k < INT32_MAX, "spmm: dimension exceeds int32");
  if (nnz > INT32_MAX)
    return fail(SB_ERR_OVERFLOW, "spmm: nnz=%lld does not fit the int32 row pointers",
                (long long)nnz);
  SB_CHECK_ARG(pos, "spmm: pos is null");
  SB_CHECK_ARG(nnz == 0 || (crd && val), "spmm: crd/val is null");
  SB_CHECK_ARG(m == 0 || k == 0 || C, "spmm: C is null");
  SB_CHECK_ARG(nnz == 0 || k == 0 || B, "spmm: B is null");
  SB_CHECK_ARG(ldb >= k && ldc >= k, "spmm: leading dimension smaller than k");
  return SB_OK;
}

template <typename T>
static int spmm_typed(int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos, const int32_t* crd, const void* val,
                      const void* B, int64_t ldb, const void* bias, int relu, int accumulate, void* C,
                      int64_t ldc, void* tile_ws, cudaStream_t st) {
  SpmmArgs<T> a = spmm_args<T>(m, n, k, nnz, pos, crd, (const T*)val, (const T*)B, ldb, (const T*)bias, relu, (T*)C,
                               ldc, 0, 0, 0);
  a.accumulate = accumulate ? 1 : 0;
  return spmm_dispatch_typed<T>(a, nnz, tile_ws, st);
}

}  // namespace sb

using namespace sb;

extern "C" {

size_t sb_spmm_csr_scratch_bytes(int64_t segments, int64_t k, int64_t batch) {
  if (segments <= 0 || k <= 0 || batch <= 0) return 0;
  // segment sums + one arrival counter per (segment, column tile of at most 256 columns)
  const size_t tiles = (size_t)ceil_div(k, 16);
  return (size_t)segments * (size_t)batch * ((size_t)k * sizeof(float) + tiles * sizeof(int));
}

static int spmm_csr_f32_impl(int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos,
                             const int32_t* crd, const float* val, const float* B, int64_t ldb,
                             const float* bias, int relu, float* C, int64_t ldc, int64_t batch,
                             int64_t stride_val, int64_t stride_b, int64_t stride_c,
                             const void* plan, int64_t plan_segments, void* scratch,
                             size_t scratch_bytes, int accumulate, void* stream) {
  int rc = check_common(m, n, k, nnz, pos, crd, val, B, ldb, C, ldc);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(batch >= 1 && batch <= 65535, "spmm: batch must be in [1, 65535]");
  SB_CHECK_ARG(stride_val >= 0 && stride_b >= 0 && stride_c >= 0, "spmm: negative batch stride");
  if (m == 0 || k == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;

  const bool vec_ok = (k % 4 == 0) && (ldb % 4 == 0) && (ldc % 4 == 0) && aligned16(B) &&
                      aligned16(C) && (!bias || aligned16(bias)) && (stride_b % 4 == 0) &&
                      (stride_c % 4 == 0) && ldb < (1ll << 32);
  if (!vec_ok && accumulate)
    return fail(SB_ERR_UNSUPPORTED,
                "spmm: accumulation needs the vector layout (k, ldb, ldc multiples of 4; B, C "
                "16-byte aligned)");
  if (plan) {
    SB_CHECK_ARG(aligned16(plan), "spmm: plan must be 16-byte aligned");
    const int64_t segs = plan_segments < 0 ? plan_cap_seg(nnz) : plan_segments;
    if (segs > 0) {
      SB_CHECK_ARG(scratch && aligned16(scratch), "spmm: scratch is null or misaligned");
      const size_t need = sb_spmm_csr_scratch_bytes(segs, k, batch);
      if (scratch_bytes < need)
        return fail(SB_ERR_WORKSPACE, "spmm: scratch has %zu bytes, needs %zu", scratch_bytes, need);
    }
  }
  // wide operands, no heavy rows: optionally the bulk-copy kernel of spmm_wide.cu
  if (k >= 512 && batch == 1 && vec_ok && !accumulate && !(plan && plan_segments != 0) && spmm_wide_wanted())
    return spmm_wide_launch(m, k, pos, crd, val, B, ldb, bias, relu, C, ldc, st);
  SpmmArgs<float> a = spmm_args<float>(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, C, ldc, stride_val,
                                       stride_b, stride_c);
  a.skip_heavy = (plan && plan_segments != 0) ? 1 : 0;
  a.accumulate = accumulate ? 1 : 0;
  return spmm_dispatch_f32(a, batch, plan, nnz, plan_segments, scratch, nullptr, st);
}

int sb_spmm_csr_f32(int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos,
                    const int32_t* crd, const float* val, const float* B, int64_t ldb,
                    const float* bias, int relu, float* C, int64_t ldc, int64_t batch,
                    int64_t stride_val, int64_t stride_b, int64_t stride_c, const void* plan,
                    int64_t plan_segments, void* scratch, size_t scratch_bytes, void* stream) {
  return spmm_csr_f32_impl(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, C, ldc, batch,
                           stride_val, stride_b, stride_c, plan, plan_segments, scratch,
                           scratch_bytes, 0, stream);
}

int sb_spmm_csr_acc_f32(int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos,
                        const int32_t* crd, const float* val, const float* B, int64_t ldb,
                        const float* bias, int relu, float* C, int64_t ldc, int64_t batch,
                        int64_t stride_val, int64_t stride_b, int64_t stride_c, const void* plan,
                        int64_t plan_segments, void* scratch, size_t scratch_bytes, void* stream) {
  return spmm_csr_f32_impl(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, C, ldc, batch,
                           stride_val, stride_b, stride_c, plan, plan_segments, scratch,
                           scratch_bytes, 1, stream);
}

size_t sb_spmm_csr_once_workspace_bytes(int dtype, int64_t k, int64_t nnz) {
  if (k <= 0 || nnz <= 0) return 16;
  return tile_workspace_bytes((dtype == SB_F64 || dtype == SB_I64) ? 8 : 4, k, nnz) + 16;
}

int sb_spmm_csr_once(int dtype, int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos,
                     const int32_t* crd, const void* val, const void* B, int64_t ldb, const void* bias,
                     int relu, int accumulate, void* C, int64_t ldc, void* ws, size_t ws_bytes,
                     void* stream) {
  int rc = check_common(m, n, k, nnz, pos, crd, val, B, ldb, C, ldc);
  if (rc != SB_OK) return rc;
  if (nnz > INT32_MAX - 4096) return fail(SB_ERR_OVERFLOW, "spmm_once: nnz=%lld does not fit int32", (long long)nnz);
  SB_CHECK_ARG(dtype >= SB_F32 && dtype <= SB_I64, "spmm_once: unknown dtype %d", dtype);
  SB_CHECK_ARG(ws && aligned16(ws), "spmm_once: workspace is null or misaligned");
  if (ws_bytes < sb_spmm_csr_once_workspace_bytes(dtype, k, nnz))
    return fail(SB_ERR_WORKSPACE, "spmm_once: workspace has %zu bytes, needs %zu", ws_bytes,
                sb_spmm_csr_once_workspace_bytes(dtype, k, nnz));
  if (m == 0 || k == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  switch (dtype) {
    case SB_F32: {
      SpmmArgs<float> a = spmm_args<float>(m, n, k, nnz, pos, crd, (const float*)val, (const float*)B, ldb,
                                           (const float*)bias, relu, (float*)C, ldc, 0, 0, 0);
      a.accumulate = accumulate ? 1 : 0;
      return spmm_dispatch_f32(a, 1, nullptr, nnz, 0, nullptr, ws, st);
    }
    case SB_F64: return spmm_typed<double>(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, accumulate, C, ldc, ws, st);
    case SB_I32:  // unsigned arithmetic: same bits as the reference's wrapping int32 math
      return spmm_typed<unsigned int>(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, accumulate, C, ldc, ws, st);
    default:
      return spmm_typed<unsigned long long>(m, n, k, nnz, pos, crd, val, B, ldb, bias, relu, accumulate, C, ldc, ws, st);
  }
}

int sb_spmm_csr_typed(int dtype, int64_t m, int64_t n, int64_t k, int64_t nnz, const int32_t* pos,
                      const int32_t* crd, const void* val, const void* B, int64_t ldb, void* C,
                      int64_t ldc, void* stream) {
  int rc = check_common(m, n, k, nnz, pos, crd, val, B, ldb, C, ldc);
  if (rc != SB_OK) return rc;
  if (m == 0 || k == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype != SB_F32 && ceil_div(k, 32) > 65535)
    return fail(SB_ERR_UNSUPPORTED, "spmm: the scalar path (dtype other than f32) takes at most %d columns, got %lld",
                65535 * 32, (long long)k);
  switch (dtype) {
    case SB_F32:
      return sb_spmm_csr_f32(m, n, k, nnz, pos, crd, (const float*)val, (const float*)B, ldb,
                             nullptr, 0, (float*)C, ldc, 1, 0, 0, 0, nullptr, 0, nullptr, 0, stream);
    case SB_F64:
      return spmm_typed<double>(m, n, k, nnz, pos, crd, val, B, ldb, nullptr, 0, 0, C, ldc, nullptr, st);
    case SB_I32:  // unsigned arithmetic: same bits as the reference's wrapping int32 math
      return spmm_typed<unsigned int>(m, n, k, nnz, pos, crd, val, B, ldb, nullptr, 0, 0, C, ldc, nullptr, st);
    case SB_I64:
      return spmm_typed<unsigned long long>(m, n, k, nnz, pos, crd, val, B, ldb, nullptr, 0, 0, C, ldc, nullptr, st);
    default:
      return fail(SB_ERR_UNSUPPORTED, "spmm_typed: unknown dtype %d", dtype);
  }
}

}  // extern "C"
