// Host check of wide_host.cpp against a CUDA runtime whose device is host
// memory: allocations can be made to fail, kernels do nothing.

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "../raycer_gb300/csrc/wide_host.cpp"

namespace
{

std::map<void*, size_t> live;            // allocations
int allocations = 0;                     // so far
int failAt = 0;                          // the allocation that fails, 0: none
cudaError_t failWith = cudaErrorMemoryAllocation;

size_t live_bytes()
{
    size_t n = 0;
    for (const auto& a : live)
        n += a.second;
    return n;
}

}  // namespace

extern "C"
{
    cudaError_t cudaMalloc(void** p, size_t n)
    {
        *p = nullptr;
        if (++allocations == failAt)
            return failWith;
        *p = std::calloc(n ? n : 1, 1);
        live[*p] = n;
        return cudaSuccess;
    }
    cudaError_t cudaFree(void* p)
    {
        if (p && live.erase(p) != 1)
            return cudaErrorInvalidValue;
        std::free(p);
        return cudaSuccess;
    }
    cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
    {
        std::memcpy(d, s, n);
        return cudaSuccess;
    }
    cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t)
    {
        return cudaMemcpy(d, s, n, k);
    }
    cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
    cudaError_t cudaGetLastError() { return cudaSuccess; }
    const char* cudaGetErrorString(cudaError_t) { return "error"; }
}

namespace rcx
{

cudaError_t launch_collapse(const DevNode*, int, WideItem*, DevNode4*, WideCounters*, int, size_t, int, cudaStream_t)
{
    return cudaSuccess;
}

}  // namespace rcx

namespace
{

int failures = 0;
#define CHECK(x)                                               \
    do                                                         \
    {                                                          \
        if (!(x))                                              \
        {                                                      \
            std::printf("line %d: %s\n", __LINE__, #x);        \
            failures++;                                        \
        }                                                      \
    } while (0)

// A tracer with a scene of `count` inner nodes.
void scene(rc_tracer& h, size_t count, int instances)
{
    h.sceneReady = true;
    h.numSMs = 4;
    h.innerCount = count;
    h.rootLink = 0;
    h.bvhDepth = 12;
    rcx::DevNode* nodes = static_cast<rcx::DevNode*>(std::calloc(count, sizeof(rcx::DevNode)));
    h.dNodes = nodes;
    h.nInstances = instances;
    h.tlasRoot = 0;
    h.tlasCount = count;
    h.dTlas = nodes;
    h.instRoots.assign(size_t(instances), 0);
}

// Without memory for a 4-wide tree a scene stays binary: no error, nothing
// left behind, and the next call neither fails nor tries again.
void allocation_failures()
{
    for (int instances : { 0, 3 })
        for (int at = 1; at <= 6; ++at)
        {
            rc_tracer h;
            scene(h, 1000, instances);
            allocations = 0;
            failAt = at;
            failWith = cudaErrorMemoryAllocation;
            CHECK(rcx::ensure_wide(&h) == RC_OK);
            CHECK(h.err.empty());
            if (instances == 0)
                CHECK(!h.dWide);
            else
                CHECK(!h.wideInstanced);
            CHECK(live_bytes() == h.deviceBytes);
            CHECK(rcx::ensure_wide(&h) == RC_OK);
            cudaFree(h.dWide);
            cudaFree(h.dWideTlas);
            cudaFree(h.dInstWide);
            CHECK(live.empty());
        }
    // another error is reported
    rc_tracer h;
    scene(h, 1000, 0);
    allocations = 0;
    failAt = 1;
    failWith = cudaErrorUnknown;
    CHECK(rcx::ensure_wide(&h) == RC_CUDA);
    CHECK(live.empty());
}

}  // namespace

int main()
{
    allocation_failures();
    if (!failures)
        std::printf("wide build ok\n");
    return failures ? 1 : 0;
}
