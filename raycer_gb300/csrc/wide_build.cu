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

#include <cuda_runtime.h>

#include <algorithm>

#include "wide_collapse.h"

namespace rcx
{
namespace
{

constexpr int kBlock = 128;

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

}  // namespace

cudaError_t launch_collapse(const DevNode* nodes, int count, WideItem* items, DevNode4* wide, WideCounters* c,
                            int level, size_t most, int numSMs, cudaStream_t stream)
{
    k_collapse_level<<<1, 1, 0, stream>>>(c, level);
    const unsigned blocks = unsigned(std::min<size_t>((most + kBlock - 1) / kBlock, size_t(numSMs) * 16));
    k_collapse<<<blocks, kBlock, 0, stream>>>(nodes, count, items, wide, c, level);
    return cudaGetLastError();
}

}  // namespace rcx
