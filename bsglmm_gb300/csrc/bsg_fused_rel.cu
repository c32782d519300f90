// bsg_fused_rel.cu -- the colour kernels of grids of up to one block per SM that let
// the next kernel in within their subject loop (REL), for the general design:
// the probit and beta_WM 16-subject step and, up to P = 5, the t/logit links.
#include "bsg_fused.cuh"

namespace bsg {
cudaError_t launch_fused_rel(int P, int threads, bool mix, bool wmu, const DatasetDev *ds,
                             ChainDev *ch, const BlockMap *map, int nblocks, int colour,
                             cudaStream_t st, bool pdl) {
  if (nblocks <= 0) return cudaSuccess;
  const Supplied sup{};
  switch (P) {
#define BSG_CASE(PP)                                                                       \
  case PP:                                                                                 \
    if (mix) {                                                                             \
      if constexpr (PP <= 5)                                                               \
        return launch_one<PP, kMixLpv, false, true, false, false, false, false, true>(      \
            nblocks, threads, st, pdl, ds, ch, map, colour, sup);                          \
      return cudaErrorInvalidValue;                                                        \
    }                                                                                      \
    return wmu ? launch_one<PP, 1, false, false, true, false, true, false, true>(           \
                     nblocks, threads, st, pdl, ds, ch, map, colour, sup)                  \
               : launch_one<PP, 1, false, false, false, false, true, false, true>(          \
                     nblocks, threads, st, pdl, ds, ch, map, colour, sup);
    BSG_CASE(1)
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
}  // namespace bsg
