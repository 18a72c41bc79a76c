// k_loops.cu -- kernels of the loop-closure segments (FP64) on the
// level-parallel driver: the tree passes on the lanes of each instance's
// group, the Gram columns on as many of them (three where the records have no
// fields for more), the multiplier solve and the projections on its first. Blocks [loopGroupFirst, +nLoopGroupBlocks) of the
// block table; records record-major (width in T.sstride). The server's blocks
// have 128 threads, a batch's one warp. 300 trees of 20 to 40 bodies, a fifth
// with closures, two steps: 13.1 ms, of which the busiest warp's FP64
// instructions are 7.5 (18.0 ms with the Gram's columns three at a time and the
// trees without closures before these instead of beside; 62.0 ms with one
// thread per instance).
#include "abi_device.cuh"

namespace sbg {

void rkLoopGroup(const KArgs& a, int threads, cudaStream_t s) {
    if (a.P->nLoopGroupBlocks <= 0) return;
    rkMersonKernel<double, 3, false, true, 1, true><<<a.P->nLoopGroupBlocks, threads, 0, s>>>(
        *a.T, a.P->loopGroupFirst, 0, a.ystate, a.time, static_cast<double*>(a.fbufLoop), a.fplane,
        static_cast<double*>(a.scratchLoop), a.status, a.h, a.step, a.accuracy, a.consTol, a.projectEveryStep);
}
void realizeLoopGroup(const KArgs& a, int threads, cudaStream_t s) {
    if (a.P->nLoopGroupBlocks <= 0) return;
    realizeKernel<double, 3, false, true, 1, true><<<a.P->nLoopGroupBlocks, threads, 0, s>>>(
        *a.T, a.P->loopGroupFirst, 0, a.y, a.ydot, static_cast<double*>(a.scratchLoop), a.status);
}
// The tree's M^-1 f (without constraints) of these instances; its records are
// field-major in the same memory.
void minvLoopGroup(const KArgs& a, int threads, cudaStream_t s) {
    if (a.P->nLoopGroupBlocks <= 0) return;
    minvKernel<double, 3, true><<<a.P->nLoopGroupBlocks, threads, 0, s>>>(
        *a.T, a.P->loopGroupFirst, 0, a.y, a.f, a.ydot, static_cast<double*>(a.scratchLoop), a.status);
}

}  // namespace sbg
