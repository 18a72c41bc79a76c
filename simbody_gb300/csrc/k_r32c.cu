// k_r32c.cu -- realize(Acceleration) kernel instantiations, FP32 recursions,
// chain driver: the dispatch and the unrefined form (the refined form is in
// k_r32cr.cu; variant 8, the staged chain driver of one shared chain
// topology, in k_r32s.cu; variant 9, the tile driver, in k_tile32.cu).
#include "r32c_launch.cuh"

namespace sbg {

void realize32Chain(const KArgs& a, bool refine, cudaStream_t s) {
    if (a.P->variant == 9)
        realizeTiles32(a, *a.tiles32, refine, a.P->chainFirst / kTile, (a.P->nChain + kTile - 1) / kTile, s);
    else if (a.P->variant == 8) realize32ChainStaged(a, refine, s);  // k_r32s.cu
    else if (refine) realize32ChainRefined(a, s);
    else r32ChainPick<false>(a, s);
}

}  // namespace sbg
