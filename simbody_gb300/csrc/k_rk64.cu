// k_rk64.cu -- fixed-step RK-Merson on the level-parallel driver, FP64: the
// serving loop's kernel (batches step on the tile driver, k_tilerk.cu).
#include "abi_device.cuh"

namespace sbg {

void rk64Group(const KArgs& a, cudaStream_t s) {
    rkMersonKernel<double, 3, false, true><<<a.P->nGroupBlocks, 128, 0, s>>>(
        *a.T, a.P->groupFirst, 0, a.ystate, a.time, static_cast<double*>(a.fbuf), a.fplane, static_cast<double*>(a.scratch), a.status,
        a.h, a.step, a.accuracy, a.consTol, a.projectEveryStep);
}

}  // namespace sbg
