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

__global__ void __launch_bounds__(kBlock) k_collapse(const DevNode* __restrict__ nodes, int count,
                                                     WideItem* __restrict__ items, DevNode4* __restrict__ wide,
                                                     WideCounters* c, int level)
{
    const int end = level_end(*c, level, count);
    for (int i = c->bound[level] + int(blockIdx.x) * kBlock + int(threadIdx.x); i < end; i += int(gridDim.x) * kBlock)
        collapse_node(nodes, count, items, wide, c, i);
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
