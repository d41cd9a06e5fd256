// Host side of the 4-wide trees' construction (kernels: wide_build.cu): which
// trees a scene gets, when, and their memory.
//
// A traversal pushes at most (children - 1) entries per node; a tree whose
// worst root-to-leaf sum exceeds the stack is left binary, and so is one for
// which there is no memory (the binary kernels serve every call), and every
// scene when RC_WIDE_BVH=0 is set in the environment (read once).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <string>
#include <vector>

#include "host_internal.h"
#include "wide_collapse.h"

namespace rcx
{
namespace
{

// A collapsed tree.
struct WideTree
{
    DevNode4* nodes = nullptr;  // null: none, the scene stays binary
    size_t count = 0;
    int need = 0;  // stack entries of a walk
};

void release(WideTree& t)
{
    cudaFree(t.nodes);
    t = WideTree{};
}

// Collapses the trees of `roots` (inner links into nodes[0, count)) into one
// array of 4-wide nodes, root i at index i. None where the stack need is above
// `maxNeed`, or where there is no memory.
rc_status collapse(rc_tracer* h, const DevNode* nodes, size_t count, const std::vector<int32_t>& roots, int levels,
                   int maxNeed, WideTree& out)
{
    WideItem* items = nullptr;
    WideCounters* counters = nullptr;
    WideCounters got{};
    std::vector<WideItem> first(roots.size());
    for (size_t i = 0; i < roots.size(); ++i)
        first[i] = WideItem{ roots[i], 0, 0, 0 };
    got.nodes = got.bound[1] = int(roots.size());
    // a wide node stands for one binary inner node
    cudaError_t e =
        cudaMalloc(reinterpret_cast<void**>(&items), count * sizeof(WideItem) + sizeof(WideCounters));
    if (e == cudaSuccess)
    {
        counters = reinterpret_cast<WideCounters*>(items + count);
        e = cudaMemcpyAsync(counters, &got, sizeof(got), cudaMemcpyHostToDevice, h->stream);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(items, first.data(), first.size() * sizeof(WideItem), cudaMemcpyHostToDevice, h->stream);
    levels = std::min(std::max(levels, 1), kMaxStack);
    for (int level = 0; e == cudaSuccess && level < levels; ++level)
    {
        // at most 4^level nodes per root
        const size_t most = level < 12 ? std::min(count, roots.size() << (2 * level)) : count;
        e = launch_collapse(nodes, int(count), items, counters, level, most, h->numSMs, h->stream);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&got, counters, sizeof(got), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(h->stream);
    const bool fits = e == cudaSuccess && !got.error && got.maxNeed <= maxNeed && got.nodes == got.bound[levels];
    if (fits)
    {
        out.count = size_t(got.nodes);
        out.need = got.maxNeed;
        e = cudaMalloc(reinterpret_cast<void**>(&out.nodes), out.count * sizeof(DevNode4));
        if (e == cudaSuccess)
            e = launch_write_nodes(nodes, items, out.nodes, got.nodes, h->stream);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(h->stream);
    }
    cudaFree(items);
    if (fits && e == cudaSuccess)
        return RC_OK;
    cudaGetLastError();
    release(out);
    if (e != cudaSuccess && e != cudaErrorMemoryAllocation)
    {
        h->err = std::string("wide BVH: ") + cudaGetErrorString(e);
        return RC_CUDA;
    }
    if (got.error)
    {
        h->err = "wide BVH: malformed binary node links";
        return RC_DEVICE_ERROR;
    }
    return RC_OK;  // stays binary
}

// The meshes' trees, the top-level one and the instances' mesh roots: all of
// them, or none.
rc_status ensure_wide_instanced(rc_tracer* h)
{
    std::vector<int32_t> roots;  // inner mesh roots, each once
    for (int32_t r : h->instRoots)
        if (r >= 0)
            roots.push_back(r);
    std::sort(roots.begin(), roots.end());
    roots.erase(std::unique(roots.begin(), roots.end()), roots.end());
    std::vector<int32_t> wideRoots;
    for (int32_t r : h->instRoots)
        wideRoots.push_back(
            r < 0 ? r : int32_t(std::lower_bound(roots.begin(), roots.end(), r) - roots.begin()));
    const int topLevels = int(h->tlasDepth);
    const int meshLevels = int(h->bvhDepth) - topLevels;
    WideTree mesh, top;
    int32_t* instWide = nullptr;
    rc_status s = RC_OK;
    bool whole = true;
    if (!roots.empty())
    {
        s = collapse(h, h->dNodes, h->innerCount, roots, meshLevels, kTwoLevelStack, mesh);
        whole = s == RC_OK && mesh.nodes;
    }
    if (whole && h->tlasRoot >= 0)
    {
        s = collapse(h, h->dTlas, h->tlasCount, { h->tlasRoot }, topLevels, kTwoLevelStack, top);
        whole = s == RC_OK && top.nodes;
    }
    // a leaf of two instances stacks its second one
    if (whole && mesh.need + top.need + 1 <= kTwoLevelStack)
    {
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&instWide), wideRoots.size() * sizeof(int32_t));
        if (e == cudaSuccess)
            e = cudaMemcpy(instWide, wideRoots.data(), wideRoots.size() * sizeof(int32_t), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
        {
            h->dWide = mesh.nodes;
            h->wideCount = mesh.count;
            h->dWideTlas = top.nodes;
            h->wideTlasCount = top.count;
            h->wideTlasRoot = h->tlasRoot >= 0 ? 0 : h->tlasRoot;
            h->dInstWide = instWide;
            h->deviceBytes += (mesh.count + top.count) * sizeof(DevNode4) + wideRoots.size() * sizeof(int32_t);
            h->wideInstanced = true;
            return RC_OK;
        }
        cudaGetLastError();
        if (e != cudaErrorMemoryAllocation)
        {
            h->err = std::string("wide BVH: ") + cudaGetErrorString(e);
            s = RC_CUDA;
        }
    }
    cudaFree(instWide);
    release(top);
    release(mesh);
    return s;
}

// Rays above the line for the 4-wide walk (cast_wide_rays) after which a scene's casts build
// its tree: what they gain by it then makes up for the construction. Measured
// with random rays (construction; k_cast -> k_cast_phased with 4M rays; rays
// for which the gain is the construction):
//   930 triangles    119 us;   611 ->   426 us; 2.6M
//   8,930            147;    1,007 ->   712;    2.0M
//   89,700           277;    1,435 ->   970;    2.4M
//   1M               574;    1,953 -> 1,250;    3.3M
//   5M               750;    2,486 -> 1,570;    3.3M
// Below the line nothing is gained (320,000 rays in 1M triangles: 340 -> 330).
constexpr int64_t kCastTreeRays = 3'000'000;

// Bounce segments, over all passes, after which a two-level scene's renders
// build its trees. A segment's launch through the binary trees takes the
// longest nested walk, whatever the paths, and that is what the trees save;
// measured at 160x90 (construction; saved per segment; segments for which the
// one is the other), and about the same at 1280x720:
//   terrain of 9,000 triangles + 3 blobs of 320         175 us;  42 us; 4.2
//   terrain of 90,000 + 40 blobs of 1,280               340;    150;    2.3
//   terrain of 90,000 + 200 blobs of 5,120              380;    240;    1.6
//   terrain of 1M + 200 blobs of 20,480                 560;    300;    1.9
constexpr int64_t kBounceTreeRounds = 4;

}  // namespace

rc_status ensure_wide_for_casts(rc_tracer* h, int64_t rays)
{
    if (h->wideTried || rays <= 0)
        return RC_OK;
    h->castRays += rays;
    return h->castRays >= kCastTreeRays ? ensure_wide(h) : RC_OK;
}

rc_status ensure_wide_for_bounces(rc_tracer* h, int64_t rounds)
{
    if (h->wideTried)
        return RC_OK;
    h->bounceRounds += rounds;
    return h->bounceRounds >= kBounceTreeRounds ? ensure_wide(h) : RC_OK;
}

rc_status ensure_wide(rc_tracer* h)
{
    if (h->wideTried || !h->sceneReady)
        return RC_OK;
    h->wideTried = true;
    h->wideRoot = h->rootLink;
    static const bool enabled = [] {
        const char* v = std::getenv("RC_WIDE_BVH");
        return !(v && v[0] == '0');
    }();
    if (!enabled)
        return RC_OK;
    if (h->nInstances > 0)
        return ensure_wide_instanced(h);
    if (h->rootLink < 0)
        return RC_OK;  // a leaf root: nothing to collapse
    WideTree tree;
    const rc_status s = collapse(h, h->dNodes, h->innerCount, { h->rootLink }, int(h->bvhDepth), kMaxStack, tree);
    if (s != RC_OK || !tree.nodes)
        return s;
    h->dWide = tree.nodes;
    h->wideCount = tree.count;
    h->wideRoot = 0;
    h->deviceBytes += h->wideCount * sizeof(DevNode4);
    return RC_OK;
}

}  // namespace rcx
