// A CUDA runtime in host memory for the host sources' tests: allocations are
// tracked, streams run in place, kernel launches do nothing, and the n-th
// allocation from now can be made to fail.
#pragma once

#include "../../psycles_b200/csrc/psy_host_internal.h"
#include "../../psycles_b200/csrc/psy_static.h"

#include <cstdlib>
#include <cstring>
#include <map>

namespace fake {
inline std::map<const void *, size_t> live;
inline int fail_in = -1;  // allocations until one fails; -1: none does
inline bool alive(const void *p) { return live.count(p) != 0u; }
inline cudaError_t allocate(void **p, size_t n) {
    if (fail_in == 0) {
        fail_in = -1;
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    if (fail_in > 0) --fail_in;
    *p = std::calloc(1, n);
    live[*p] = n;
    return cudaSuccess;
}
inline cudaError_t release(void *p) {
    live.erase(p);
    std::free(p);
    return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { return fake::allocate(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return fake::allocate(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return fake::allocate(p, n); }
cudaError_t cudaFree(void *p) { return fake::release(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaFreeHost(void *p) { return fake::release(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(8);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = reinterpret_cast<cudaEvent_t>(8);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

namespace psy {
void launch_bake_materials(cudaStream_t, const SceneView &, BakedMaterialGpu *, BakedClosureGpu *, uint32_t, uint32_t) {}
void launch_pack_triangles(cudaStream_t, const MeshGpu *, uint32_t, const float *, const float *, const uint32_t *,
                           const uint32_t *, const uint32_t *, uint32_t, TriGpu *, ShadeTriGpu *) {}
}  // namespace psy
