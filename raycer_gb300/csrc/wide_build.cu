// 4-wide BVHs, collapsed on the device from a scene's binary nodes at its
// first use by a kernel that walks them: the tree of a single-level scene, or
// the trees of a two-level scene's meshes and the one over its instances.
//
// Each wide node starts from one binary node's two children and repeatedly
// replaces its inner child of largest surface area by that child's two
// children, up to four. Leaves stay as they are (the same triangles in the
// same order), so a triangle test of the wide traversal is the binary
// traversal's. A child box of the binary tree lies inside its parent's box
// (also in float: both were rounded to nearest from nested boxes, or are
// float unions), and the slab test is monotone in the box, so every ray that
// reaches a grandchild through the binary tree reaches it through the wide
// node too: the nearest-first closest hit, which does not depend on the
// visiting order, is the same.
//
// One launch per level: thread i takes the i-th wide node of the level,
// chooses its children and takes consecutive nodes of the next level for the
// inner ones (one atomic). What bounds it is the chain of levels, two
// launches each. A scene's first PATH frame, the collapse included (on the
// host before: nodes downloaded, collapsed, uploaded): 1M triangles
// 10.6 -> 2.3 ms, 5M triangles 67.8 -> 5.7 ms.
//
// The traversal pushes at most (children - 1) entries per node; a tree whose
// worst root-to-leaf sum exceeds the stack is left binary, and so is every
// scene when RC_WIDE_BVH=0 is set in the environment (read once).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <string>
#include <vector>

#include "host_internal.h"

namespace rcx
{
namespace
{

constexpr int kBlock = 128;

// Counters of a collapse (device memory). Level l's nodes are
// [bound[l], bound[l + 1]).
struct WideCounters
{
    int nodes;    // wide nodes taken
    int maxNeed;  // stack entries pushed on the worst root-to-leaf path
    int error;    // malformed binary links
    int bound[kMaxStack + 2];
};

// What a wide node is made from.
struct WideItem
{
    int bin;   // its binary inner node
    int need;  // stack entries pushed above it
};

struct Child
{
    int link;
    float lo[3];
    float hi[3];
};

__device__ __forceinline__ void children_of(const DevNode& n, Child& a, Child& b)
{
    a = Child{ n.link.x, { n.xy0.x, n.xy0.z, n.z01.x }, { n.xy0.y, n.xy0.w, n.z01.y } };
    b = Child{ n.link.y, { n.xy1.x, n.xy1.z, n.z01.z }, { n.xy1.y, n.xy1.w, n.z01.w } };
}

__device__ __forceinline__ float half_area(const Child& c)
{
    const float dx = fmaxf(0.0f, c.hi[0] - c.lo[0]);
    const float dy = fmaxf(0.0f, c.hi[1] - c.lo[1]);
    const float dz = fmaxf(0.0f, c.hi[2] - c.lo[2]);
    return dx * dy + dy * dz + dz * dx;
}

__global__ void __launch_bounds__(kBlock) k_collapse(const DevNode* __restrict__ nodes, int count,
                                                     WideItem* __restrict__ items, DevNode4* __restrict__ wide,
                                                     WideCounters* c, int level)
{
    const int end = c->bound[level + 1];
    for (int i = c->bound[level] + int(blockIdx.x) * kBlock + int(threadIdx.x); i < end; i += int(gridDim.x) * kBlock)
    {
        const WideItem it = items[i];
        Child ch[4];
        int n = 2;
        children_of(nodes[it.bin], ch[0], ch[1]);
        bool bad = false;
        while (n < 4)
        {
            int best = -1;
            float bestA = -1.0f;
            for (int k = 0; k < n; ++k)
                if (ch[k].link >= 0 && half_area(ch[k]) > bestA)
                {
                    best = k;
                    bestA = half_area(ch[k]);
                }
            if (best < 0)
                break;
            if (ch[best].link >= count)
            {
                bad = true;
                break;
            }
            Child x, y;
            children_of(nodes[ch[best].link], x, y);
            ch[best] = x;
            ch[n++] = y;
        }
        int inner = 0;
        for (int k = 0; k < n; ++k)
        {
            if (ch[k].link >= count)
                bad = true;
            if (ch[k].link >= 0)
                inner++;
        }
        int node = bad ? 0 : atomicAdd(&c->nodes, inner);
        if (bad || node + inner > count)
        {
            c->error = 1;  // links that are no tree
            continue;
        }
        const int need = it.need + (n - 1);
        atomicMax(&c->maxNeed, need);
        DevNode4 w{};
        float* lox = &w.lox.x;
        float* hix = &w.hix.x;
        float* loy = &w.loy.x;
        float* hiy = &w.hiy.x;
        float* loz = &w.loz.x;
        float* hiz = &w.hiz.x;
        int* link = &w.link.x;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            if (k >= n)
                break;
            lox[k] = ch[k].lo[0];
            hix[k] = ch[k].hi[0];
            loy[k] = ch[k].lo[1];
            hiy[k] = ch[k].hi[1];
            loz[k] = ch[k].lo[2];
            hiz[k] = ch[k].hi[2];
            if (ch[k].link >= 0)
            {
                items[node] = WideItem{ ch[k].link, need };
                link[k] = node++;
                continue;
            }
            link[k] = ch[k].link;
        }
        w.meta.x = n;
        wide[i] = w;
    }
}

// Closes the level just taken.
__global__ void k_collapse_level(WideCounters* c, int level) { c->bound[level + 1] = c->nodes; }

// Collapses the trees of `roots` (inner links into nodes[0, count)) into one
// array of 4-wide nodes, root i at index i. *out stays null where the stack
// need (*need) is above `maxNeed`.
rc_status collapse(rc_tracer* h, const DevNode* nodes, size_t count, const std::vector<int32_t>& roots, int levels,
                   int maxNeed, DevNode4** out, int* need)
{
    *out = nullptr;
    WideItem* items = nullptr;
    WideCounters* counters = nullptr;
    WideCounters got{};
    std::vector<WideItem> first(roots.size());
    for (size_t i = 0; i < roots.size(); ++i)
        first[i] = WideItem{ roots[i], 0 };
    got.nodes = int(roots.size());
    // a wide node stands for one binary inner node
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(out), count * sizeof(DevNode4));
    if (e == cudaSuccess)
        e = cudaMalloc(reinterpret_cast<void**>(&items), count * sizeof(WideItem) + sizeof(WideCounters));
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
        k_collapse_level<<<1, 1, 0, h->stream>>>(counters, level);
        // at most 4^level nodes per root
        const size_t most = level < 12 ? std::min(count, roots.size() << (2 * level)) : count;
        const unsigned blocks = unsigned(std::min<size_t>((most + kBlock - 1) / kBlock, size_t(h->numSMs) * 16));
        k_collapse<<<blocks, kBlock, 0, h->stream>>>(nodes, int(count), items, *out, counters, level);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&got, counters, sizeof(got), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(h->stream);
    cudaFree(items);
    if (e == cudaSuccess && !got.error && got.maxNeed <= maxNeed && got.nodes == got.bound[levels])
    {
        *need = got.maxNeed;
        return RC_OK;
    }
    cudaGetLastError();
    cudaFree(*out);
    *out = nullptr;
    if (e != cudaSuccess)
    {
        h->err = std::string("wide BVH: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? RC_OOM : RC_CUDA;
    }
    if (got.error)
    {
        h->err = "wide BVH: malformed binary node links";
        return RC_DEVICE_ERROR;
    }
    return RC_OK;  // stays binary
}

// The meshes' trees, the top-level one and the instances' mesh roots.
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
    const int levels = int(std::min<uint64_t>(h->bvhDepth, kMaxStack));
    int needMesh = 0, needTop = 0;
    rc_status s = RC_OK;
    if (!roots.empty() &&
        ((s = collapse(h, h->dNodes, h->innerCount, roots, levels, kTwoLevelStack, &h->dWide, &needMesh)) != RC_OK ||
         !h->dWide))
        return s;
    h->wideCount = h->dWide ? h->innerCount : 0;
    h->deviceBytes += h->wideCount * sizeof(DevNode4);
    h->wideTlasRoot = h->tlasRoot;
    if (h->tlasRoot >= 0)
    {
        s = collapse(h, h->dTlas, h->tlasCount, { h->tlasRoot }, levels, kTwoLevelStack, &h->dWideTlas, &needTop);
        if (s != RC_OK || !h->dWideTlas)
            return s;
        h->wideTlasRoot = 0;
        h->wideTlasCount = h->tlasCount;
        h->deviceBytes += h->wideTlasCount * sizeof(DevNode4);
    }
    // a leaf of two instances stacks its second one
    if (needMesh + needTop + 1 > kTwoLevelStack)
        return RC_OK;  // stays binary
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&h->dInstWide), wideRoots.size() * sizeof(int32_t));
    if (e == cudaSuccess)
    {
        h->deviceBytes += wideRoots.size() * sizeof(int32_t);
        e = cudaMemcpy(h->dInstWide, wideRoots.data(), wideRoots.size() * sizeof(int32_t), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess)
    {
        cudaGetLastError();
        h->err = std::string("wide BVH: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? RC_OOM : RC_CUDA;
    }
    h->wideInstanced = true;
    return RC_OK;
}

}  // namespace

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
    int need = 0;
    const rc_status s = collapse(h, h->dNodes, h->innerCount, { h->rootLink }, int(h->bvhDepth), kMaxStack, &h->dWide,
                                 &need);
    if (s != RC_OK || !h->dWide)
        return s;
    h->wideCount = h->innerCount;
    h->wideRoot = 0;
    h->deviceBytes += h->wideCount * sizeof(DevNode4);
    return RC_OK;
}

}  // namespace rcx
