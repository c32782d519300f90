// bsg_fused_one_wide.cu -- instantiations of the fused colour kernel for studies
// whose first design column is all ones (one lane per voxel, Philox variates),
// on the 16-subject step, with and without the beta_WM update.
#include "bsg_fused.cuh"

namespace bsg {
namespace {
template <bool WMU>
cudaError_t go(int P, int threads, const DatasetDev *ds, ChainDev *ch, const BlockMap *map,
               int nblocks, int colour, cudaStream_t st, bool pdl) {
  const Supplied sup{};
  switch (P) {
#define BSG_CASE(PP)                                                                     \
  case PP:                                                                               \
    return launch_one<PP, 1, false, false, WMU, false, true, true>(                      \
        nblocks, threads, st, pdl, ds, ch, map, colour, sup);
    BSG_CASE(2)
    BSG_CASE(3)
    BSG_CASE(4)
    BSG_CASE(5)
    BSG_CASE(6)
    BSG_CASE(7)
    BSG_CASE(8)
#undef BSG_CASE
    default:
      return cudaErrorInvalidValue;
  }
}
}  // namespace

cudaError_t launch_fused_one_wide(int P, int threads, bool wmu, const DatasetDev *ds,
                                  ChainDev *ch, const BlockMap *map, int nblocks, int colour,
                                  cudaStream_t st, bool pdl) {
  if (nblocks <= 0) return cudaSuccess;
  return wmu ? go<true>(P, threads, ds, ch, map, nblocks, colour, st, pdl)
             : go<false>(P, threads, ds, ch, map, nblocks, colour, st, pdl);
}

}  // namespace bsg
