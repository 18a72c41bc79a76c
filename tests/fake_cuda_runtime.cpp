// A CUDA runtime without a GPU, for tests of the host side (capi.cpp) on the
// CPU: device memory is host memory, kernels do nothing, and an asynchronous
// copy takes place when its stream is waited for, so that a copy still under
// way when a call returns can be seen. Any call can be made to fail.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <set>
#include <vector>

#include "../simbody_gb300/csrc/kernels.h"

namespace {

struct Stream;
struct Event {
    Stream* s = nullptr;
    size_t upto = 0;
};
struct Op {
    std::function<void()> run;
    bool copy;
};
struct Stream {
    std::vector<Op> ops;
    size_t done = 0;
    void flush(size_t upto) {
        while (done < upto && done < ops.size()) ops[done++].run();
    }
};
std::set<Stream*> streams;
std::set<const void*> pinned;
int pageable = 1;
long calls = 0, failAt = 0;  // the failAt-th call that may fail does (0: none)

cudaError_t check() { return failAt && ++calls == failAt ? cudaErrorUnknown : cudaSuccess; }
Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
Event* of(cudaEvent_t e) { return reinterpret_cast<Event*>(e); }

}  // namespace

extern "C" {

void fake_pageable(int on) { pageable = on; }
// The n-th call from now on fails (0: none); returns how many were made since.
long fake_fail_at(long n) {
    const long made = calls;
    calls = 0;
    failAt = n;
    return made;
}
long fake_calls() { return calls; }
int fake_copies_under_way() {
    int n = 0;
    for (Stream* s : streams)
        for (size_t k = s->done; k < s->ops.size(); ++k) n += s->ops[k].copy;
    return n;
}

#define MAY_FAIL()                                      \
    do {                                                \
        if (check() != cudaSuccess) return cudaErrorUnknown; \
    } while (0)

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { MAY_FAIL(); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 4 : pageable;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { MAY_FAIL(); *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { MAY_FAIL(); *p = std::calloc(1, n ? n : 1); pinned.insert(*p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { pinned.erase(p); std::free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = pinned.count(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    MAY_FAIL();
    Stream* n = new Stream;
    streams.insert(n);
    *s = reinterpret_cast<cudaStream_t>(n);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { streams.erase(of(s)); delete of(s); return cudaSuccess; }
// A failed wait has not waited, the first time; the copies take place at the next one.
cudaError_t cudaStreamSynchronize(cudaStream_t s) { MAY_FAIL(); of(s)->flush(of(s)->ops.size()); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { MAY_FAIL(); *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete of(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    MAY_FAIL();
    of(e)->s = of(s);
    of(e)->upto = of(s)->ops.size();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    MAY_FAIL();
    const Event at = *of(e);
    of(s)->ops.push_back({[at] { if (at.s) at.s->flush(at.upto); }, false});
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { MAY_FAIL(); if (of(e)->s) of(e)->s->flush(of(e)->upto); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    MAY_FAIL();
    of(st)->ops.push_back({[=] { std::memcpy(d, s, n); }, true});
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { MAY_FAIL(); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { MAY_FAIL(); std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    MAY_FAIL();
    of(st)->ops.push_back({[=] { std::memset(d, v, n); }, false});
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { MAY_FAIL(); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = reinterpret_cast<cudaGraphExec_t>(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { MAY_FAIL(); return cudaSuccess; }

}  // extern "C"

namespace sbg {
// Only the host side is under test; the kernels' results are not looked at.
cudaError_t launchRealize(const DevTables&, const LaunchPlan&, int, const double*, double*, const BatchBufs&, int32_t*, const Streams&) { return check(); }
cudaError_t launchMInv(const DevTables&, const LaunchPlan&, int, const double*, const double*, double*, const BatchBufs&, int32_t*, const Streams&) { return check(); }
cudaError_t launchRKMerson(const DevTables&, const LaunchPlan&, int, double*, double*, const BatchBufs&, int32_t*, double, StepCtl, double, double, int, const Streams&) { return check(); }
cudaError_t launchTreeOp(const DevTables&, const LaunchPlan&, const TileSet&, const OpIO&, const double*, double*, int32_t*, cudaStream_t) { return check(); }
cudaError_t launchNormalizeQuat(const DevTables&, double*, cudaStream_t) { return check(); }
cudaError_t launchQDotDot(const DevTables&, const int64_t*, const double*, const double*, double*, cudaStream_t) { return check(); }
cudaError_t launchScatter(const Packing&, const int64_t*, const double*, double*, int, cudaStream_t, int, int) { return check(); }
cudaError_t launchGather(const Packing&, const int64_t*, const double*, double*, int, cudaStream_t, int, int) { return check(); }
cudaError_t launchRKFp64List(const DevTables&, const TileSet&, const TileSet&, double*, double*, int32_t*, double, StepCtl, double, double, int, int64_t, cudaStream_t) { return check(); }
cudaError_t launchTilePar(const DevTables&, const int32_t*, int64_t, int, double*, cudaStream_t) { return check(); }
cudaError_t launchFillInt(int32_t*, int, int, cudaStream_t) { return check(); }
cudaError_t launchCountUnfinished(int, const int32_t*, const double*, const int32_t*, double, int32_t*, cudaStream_t) { return check(); }
void realizeTiles(const KArgs&, const TileSet&, int, int, cudaStream_t) {}
void realize32Chain(const KArgs&, bool, cudaStream_t) {}
void realizeFallbackTiles(const KArgs&, const TileSet&, int, int, const TileSet&, int, int, int, int, cudaStream_t) {}
void rkAdaptiveTiles(const KArgs&, const TileSet&, const AdaptCtl&, cudaStream_t) {}
}  // namespace sbg
