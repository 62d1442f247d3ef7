// SpMM forms of the other value types: float64 with 32, 16 and 8 byte loads, the integers with one
// element per load.
#include "spmm_kernels.cuh"
#include "spmm_tiles.cuh"

namespace sb {

template <typename T>
int spmm_dispatch_typed(const SpmmArgs<T>& a, int64_t nnz, void* tile_ws, cudaStream_t st) {
  void* const scratch = nullptr;
  constexpr int64_t batch = 1, plan_segments = 0;
  constexpr const void* plan = nullptr;
  const int k = a.k;
  if constexpr (std::is_same<T, double>::value) {
    const unsigned align = spmm_alignment(a);
    if (a.ldb < (1ll << 32) && align == 32) {
      if (k <= 16) SB_GO(4, 1, 4, false);
      if (k <= 32) SB_GO(8, 1, 4, false);
      if (k <= 64) SB_GO(16, 1, 4, false);
      SB_GO(32, 1, 4, false);
    }
    if (a.ldb < (1ll << 32) && align == 16) {
      if (k <= 8) SB_GO(4, 1, 2, false);
      if (k <= 16) SB_GO(8, 1, 2, false);
      if (k <= 32) SB_GO(16, 1, 2, false);
      if (k <= 64) SB_GO(32, 1, 2, false);
      SB_GO(32, 2, 2, false);
    }
  }
  if (k <= 4) SB_GO(4, 1, 1, false);
  if (k <= 16) SB_GO(16, 1, 1, false);
  if (k <= 32) SB_GO(32, 1, 1, false);
  SB_GO(32, 3, 1, false);
}

template int spmm_dispatch_typed<double>(const SpmmArgs<double>&, int64_t, void*, cudaStream_t);
template int spmm_dispatch_typed<unsigned int>(const SpmmArgs<unsigned int>&, int64_t, void*, cudaStream_t);
template int spmm_dispatch_typed<unsigned long long>(const SpmmArgs<unsigned long long>&, int64_t, void*,
                                                     cudaStream_t);

}  // namespace sb
