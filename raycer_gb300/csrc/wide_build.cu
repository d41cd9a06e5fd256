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
// float unions), and the slab test is monotone in the box where it meets no
// NaN, so every ray that reaches a grandchild through the binary tree reaches it
// through the wide node too, and no other: the nearest-first closest hit is the
// same (traverse.cuh says for which rays it is not, and what they do).
//
// One launch per level: thread i takes the i-th wide node of the level,
// chooses its children and takes consecutive nodes of the next level for the
// inner ones (one atomic). The nodes are written once their number is known,
// into an array of just that many (111,096 for the 275,270 binary nodes of
// 1M triangles of terrain). What bounds it is the chain of levels. A scene's
// first PATH frame, the collapse included (on the host before: nodes
// downloaded, collapsed, uploaded): 1M triangles 10.6 -> 2.3 ms, 5M triangles
// 67.8 -> 5.7 ms.

#include <cuda_runtime.h>

#include <algorithm>

#include "wide_collapse.h"

namespace rcx
{
namespace
{

constexpr int kBlock = 128;

// Takes a level's nodes; the last block closes the level they go to.
__global__ void __launch_bounds__(kBlock) k_collapse(const DevNode* __restrict__ nodes, int count,
                                                     WideItem* __restrict__ items, WideCounters* c, int level)
{
    const int end = level_end(*c, level, count);
    for (int i = c->bound[level] + int(blockIdx.x) * kBlock + int(threadIdx.x); i < end; i += int(gridDim.x) * kBlock)
        collapse_node(nodes, count, items, c, i);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(&c->blocks[level], 1) == int(gridDim.x) - 1)
            c->bound[level + 2] = atomicAdd(&c->nodes, 0);
    }
}

__global__ void __launch_bounds__(kBlock) k_write_nodes(const DevNode* __restrict__ nodes,
                                                        const WideItem* __restrict__ items,
                                                        DevNode4* __restrict__ wide, int taken)
{
    const int i = int(blockIdx.x) * kBlock + int(threadIdx.x);
    if (i < taken)
        write_node(nodes, items, wide, i);
}

}  // namespace

cudaError_t launch_collapse(const DevNode* nodes, int count, WideItem* items, WideCounters* c, int level, size_t most,
                            int numSMs, cudaStream_t stream)
{
    const unsigned blocks = unsigned(std::min<size_t>((most + kBlock - 1) / kBlock, size_t(numSMs) * 16));
    k_collapse<<<blocks, kBlock, 0, stream>>>(nodes, count, items, c, level);
    return cudaGetLastError();
}

cudaError_t launch_write_nodes(const DevNode* nodes, const WideItem* items, DevNode4* wide, int taken,
                               cudaStream_t stream)
{
    k_write_nodes<<<unsigned((taken + kBlock - 1) / kBlock), kBlock, 0, stream>>>(nodes, items, wide, taken);
    return cudaGetLastError();
}

}  // namespace rcx
