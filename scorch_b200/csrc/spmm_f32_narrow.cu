// fp32 SpMM forms for operands whose rows are aligned to 8 or 4 bytes only (a width that is no
// multiple of 4, column slices at odd offsets).
//
// Bound by L2 -> SM gathers like the aligned forms, with more load instructions per byte: a warp
// spans the row with 32 lanes x VEC one- or two-element loads, so a 77-column row is three
// coalesced 128-byte requests.  70,001 rows, 20 entries each, 77 columns: 3.54 ms with the former
// lane-per-column loop, which walked every row in one serial chain.
#include "spmm_kernels.cuh"
#include "spmm_tiles.cuh"

namespace sb {

int spmm_dispatch_f32_narrow(const SpmmArgs<float>& a, int64_t batch, const void* plan, int64_t nnz,
                             int64_t plan_segments, void* scratch, void* tile_ws, cudaStream_t st) {
  using T = float;
  const int k = a.k;
  if (spmm_alignment(a) >= 8 && a.ldb < (1ll << 32)) {
    if (k <= 8) SB_GO(4, 1, 2, false);
    if (k <= 16) SB_GO(8, 1, 2, false);
    if (k <= 32) SB_GO(16, 1, 2, false);
    // as few panels of at most 256 columns as the width needs, of equal width
    switch (ceil_div(ceil_div(k, 64), ceil_div(k, 256))) {
      case 1: SB_GO(32, 1, 2, false);
      case 2: SB_GO(32, 2, 2, false);
      case 3: SB_GO(32, 3, 2, false);
      default: SB_GO(32, 4, 2, false);
    }
  }
  if (k <= 4) SB_GO(4, 1, 1, false);
  if (k <= 8) SB_GO(8, 1, 1, false);
  if (k <= 16) SB_GO(16, 1, 1, false);
  switch (ceil_div(ceil_div(k, 32), ceil_div(k, 128))) {
    case 1: SB_GO(32, 1, 1, false);
    case 2: SB_GO(32, 2, 1, false);
    case 3: SB_GO(32, 3, 1, false);
    default: SB_GO(32, 4, 1, false);
  }
}

}  // namespace sb
