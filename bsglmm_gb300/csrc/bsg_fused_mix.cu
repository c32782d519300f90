// bsg_fused_mix.cu -- instantiations of the fused colour kernel for the
// t/logit links (two lanes per voxel, Philox variates): with X' Phi X in
// registers the kernel fits two 256-thread blocks per SM up to P = 5, and two
// lanes per voxel make the brain-sized grid about three full waves instead of
// 1.5.  Above P = 5 it comes in two forms: blocks of up to 128 threads, three
// per SM at 168 registers, and one of 256 at 206 or so, which is better only
// where the grid fills each SM just once.  us per sweep, one block of 256 /
// three of 128, logistic: 84,368 voxels N = 251 P = 6 473 / 342, 290,369 voxels
// N = 60 P = 8 833 / 680, 38,456 voxels (151 blocks of 256) N = 1200 P = 6
// 525 / 608.
#include "bsg_fused.cuh"

namespace bsg {
namespace {
template <int P>
cudaError_t launch_mix(int nblocks, int threads, const DatasetDev *ds, ChainDev *ch,
                       const BlockMap *map, int colour, cudaStream_t st, bool pdl) {
  const Supplied sup{};
  if constexpr (P > 5)
    if (threads <= kSmallBlock)
      return launch_one<P, kMixLpv, false, true, false, false, true, false>(
          nblocks, threads, st, pdl, ds, ch, map, colour, sup);
  return launch_one<P, kMixLpv, false, true, false, false, false, false>(
      nblocks, threads, st, pdl, ds, ch, map, colour, sup);
}
}  // namespace

cudaError_t launch_fused_mix(int P, int threads, const DatasetDev *ds, ChainDev *ch,
                     const BlockMap *map, int nblocks, int colour, cudaStream_t st,
                     bool pdl) {
  if (nblocks <= 0) return cudaSuccess;
  switch (P) {
    case 1: return launch_mix<1>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 2: return launch_mix<2>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 3: return launch_mix<3>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 4: return launch_mix<4>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 5: return launch_mix<5>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 6: return launch_mix<6>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 7: return launch_mix<7>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 8: return launch_mix<8>(nblocks, threads, ds, ch, map, colour, st, pdl);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace bsg
