// bsg_fused_mix_one.cu -- the instantiations of bsg_fused_mix.cu for studies
// whose first design column is all ones, up to P = 5 (two loads less per subject
// at P = 5: logistic, N = 301, 637 -> 622 us per sweep; above, the form for
// blocks of 128 threads loses 1 to 4 % by it).
#include "bsg_fused.cuh"

namespace bsg {
namespace {
template <int P>
cudaError_t launch_mix(int nblocks, int threads, const DatasetDev *ds, ChainDev *ch,
                       const BlockMap *map, int colour, cudaStream_t st, bool pdl) {
  const Supplied sup{};
  return launch_one<P, kMixLpv, false, true, false, false, false, true>(
      nblocks, threads, st, pdl, ds, ch, map, colour, sup);
}
}  // namespace

cudaError_t launch_fused_mix_one(int P, int threads, const DatasetDev *ds, ChainDev *ch,
                                 const BlockMap *map, int nblocks, int colour,
                                 cudaStream_t st, bool pdl) {
  if (nblocks <= 0) return cudaSuccess;
  switch (P) {
    case 2: return launch_mix<2>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 3: return launch_mix<3>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 4: return launch_mix<4>(nblocks, threads, ds, ch, map, colour, st, pdl);
    case 5: return launch_mix<5>(nblocks, threads, ds, ch, map, colour, st, pdl);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace bsg
