// steps_device.cuh -- step-size and step-list logic shared by the RK-Merson
// kernels of both drivers.
#pragma once
#include "kernels.h"

namespace sbg {

// takeOneStep's choice of the step's end against tMax = tStop
// (AbstractIntegratorRep.cpp:536-544). False: tStop is reached, or time no
// longer advances.
__device__ __forceinline__ bool stepToTarget(double tc, double h, double tStop, double* t1) {
    if (!(tc < tStop)) return false;
    if (tStop < tc + 0.95 * h) *t1 = tStop;
    else if (tStop > tc + 1.001 * h) *t1 = tc + h;
    else *t1 = tStop;
    return *t1 > tc;
}

// q slots of a body by its info word (Ball and Free keep the quaternion's).
__device__ __forceinline__ int slotQ(int info) {
    const int type = info & 15;
    return type == SBG_BALL ? 4 : type == SBG_FREE ? 7 : (info >> 4) & 15;
}

// One-step launches of a mixed batch integration: the instance's mode at the
// next launch (written by this launch's owner of the instance only); FP64
// puts it on the next list.
__device__ __forceinline__ void fbNext(const DevTables& T, int launch, int inst, bool fp64) {
    const int k = (launch + 1) & 1;
    T.fbMode[(int64_t)k * T.ninst + inst] = fp64 ? 1 : 0;
    if (fp64) T.fbList[(int64_t)k * T.ninst + atomicAdd(T.fbCount + k, 1)] = inst;
}

}  // namespace sbg
