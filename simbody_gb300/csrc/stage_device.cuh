// stage_device.cuh -- a body's record fields staged through shared memory by
// cp.async, for the drivers whose 32 instances of a warp share a scratch tile:
// the staged chain driver (k_r32s.cu) and the FP32 tile driver
// (tile32_device.cuh).
#pragma once
#include "abi_device.cuh"

namespace sbg {

// A pass's read set: up to four field ranges, packed in this order in the
// shared buffer (slot s holds the 32 lanes' values of one field).
template <int A0, int A1, int B0, int B1, int C0, int C1, int D0, int D1> struct StageSet {
    static constexpr int nA = A1 - A0, nB = B1 - B0, nC = C1 - C0, nD = D1 - D0;
    static constexpr int size = nA + nB + nC + nD;
    static __device__ __forceinline__ constexpr int slot(int f) {
        return (f >= A0 && f < A1) ? f - A0
               : (f >= B0 && f < B1) ? nA + f - B0
               : (f >= C0 && f < C1) ? nA + nB + f - C0
               : (f >= D0 && f < D1) ? nA + nB + nC + f - D0
                                     : -1;
    }
};

template <int N> struct Sets {
    static constexpr int ef = kRecH + 6 * N, eDI = ef + N, eG = eDI + N * N, eEps = eG + 6 * N, eU0 = eEps + N,
                         end = eU0 + N;
    using P2 = StageSet<kRecPc, kRecBF + 6, kRecH, eDI, 0, 0, 0, 0>;
    using P3 = StageSet<kRecH, eU0, 0, 0, 0, 0, 0, 0>;
    using P4 = StageSet<kRecL, kRecL + 3, kRecFdf, kRecFdf + 12, kRecH, eDI, eG, eEps>;
    using P5 = StageSet<kRecL, kRecL + 3, kRecH, ef, eDI, end, 0, 0>;
    static constexpr int maxSize = P2::size > P3::size ? (P2::size > P4::size ? (P2::size > P5::size ? P2::size : P5::size)
                                                                               : (P4::size > P5::size ? P4::size : P5::size))
                                                       : (P3::size > P4::size ? (P3::size > P5::size ? P3::size : P5::size)
                                                                               : (P4::size > P5::size ? P4::size : P5::size));
};

// Element f of the current record: from the shared buffer when the pass
// staged it, else from the lane's column of the tile in global memory.
template <class SET> struct ScrStaged {
    float* g;   // lane's column of the tile: element (rec + f) * 32
    float* sm;  // lane's column of the current buffer: slot s at s * 32
    __device__ __forceinline__ float& operator()(int rec, int f) const {
        const int s = SET::slot(f);
        return s >= 0 ? sm[s * kTile] : g[(rec + f) * kTile];
    }
};

__device__ __forceinline__ void cpAsync16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void prefetchL2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K> __device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

// Copy fields [F0, F1) of the record at recTile (the tile's element of
// field 0 of the record) to slots [S0, ...) of the buffer at byte address sbuf.
template <int F0, int F1, int S0>
__device__ __forceinline__ void stageRange(const float* recTile, uint32_t sbuf, int lane) {
    constexpr int chunks = (F1 - F0) * (kTile / 4);  // 16-byte chunks
#pragma unroll 4
    for (int c = lane; c < chunks; c += 32)
        cpAsync16(sbuf + (uint32_t)((S0 * kTile + 4 * c) * 4), recTile + F0 * kTile + 4 * c);
}
template <class SET, int A0, int A1, int B0, int B1, int C0, int C1, int D0, int D1>
__device__ __forceinline__ void stageAll(StageSet<A0, A1, B0, B1, C0, C1, D0, D1>*, const float* recTile, uint32_t sbuf,
                                         int lane) {
    if constexpr (A1 > A0) stageRange<A0, A1, 0>(recTile, sbuf, lane);
    if constexpr (B1 > B0) stageRange<B0, B1, SET::nA>(recTile, sbuf, lane);
    if constexpr (C1 > C0) stageRange<C0, C1, SET::nA + SET::nB>(recTile, sbuf, lane);
    if constexpr (D1 > D0) stageRange<D0, D1, SET::nA + SET::nB + SET::nC>(recTile, sbuf, lane);
}
template <class SET> __device__ __forceinline__ void stage(const float* recTile, uint32_t sbuf, int lane) {
    stageAll<SET>(static_cast<SET*>(nullptr), recTile, sbuf, lane);
}

}  // namespace sbg
