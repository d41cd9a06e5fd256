// Records, per-node steps and launches of the 4-wide trees' construction: the
// kernels are in wide_build.cu, the host side in wide_host.cpp. Links that are
// no tree (an index outside the nodes, more nodes than there are) are found
// before they are followed, and set `error`.
#pragma once

#include <cuda_runtime.h>

#include <math.h>

#include "device_types.h"

namespace rcx
{

// Counters of a collapse (device memory). Level l's nodes are
// [bound[l], bound[l + 1]).
struct WideCounters
{
    int nodes;    // wide nodes taken
    int maxNeed;  // stack entries pushed on the worst root-to-leaf path
    int error;    // malformed binary links
    int bound[kMaxStack + 2];
    int blocks[kMaxStack];  // blocks of the level's launch that are done
};

// What a wide node is made from.
struct WideItem
{
    int bin;     // its binary inner node
    int need;    // stack entries pushed above it
    int child;   // its first inner child; the others follow
    int opened;  // the children opened, 4 bits each (index + 1), in order
};

struct WideChild
{
    int link;
    float lo[3];
    float hi[3];
};

__host__ __device__ inline void children_of(const DevNode& n, WideChild& a, WideChild& b)
{
    a = WideChild{ n.link.x, { n.xy0.x, n.xy0.z, n.z01.x }, { n.xy0.y, n.xy0.w, n.z01.y } };
    b = WideChild{ n.link.y, { n.xy1.x, n.xy1.z, n.z01.z }, { n.xy1.y, n.xy1.w, n.z01.w } };
}

__host__ __device__ inline double half_area(const WideChild& c)
{
    const double dx = fmax(0.0, double(c.hi[0]) - double(c.lo[0]));
    const double dy = fmax(0.0, double(c.hi[1]) - double(c.lo[1]));
    const double dz = fmax(0.0, double(c.hi[2]) - double(c.lo[2]));
    return dx * dy + dy * dz + dz * dx;
}

// Replaces child `k` of n by its own children.
__host__ __device__ inline void open_child(const DevNode* nodes, WideChild* ch, int& n, int k)
{
    WideChild x, y;
    children_of(nodes[ch[k].link], x, y);
    ch[k] = x;
    ch[n++] = y;
}

// Children of the wide node of binary node `bin`, and how many: 2 to 4, or 0
// where a link is no index of the `count` nodes; the ones opened in `opened`.
__host__ __device__ inline int wide_children(const DevNode* nodes, int count, int bin, WideChild* ch, int& opened)
{
    opened = 0;
    if (bin < 0 || bin >= count)
        return 0;
    int n = 2;
    children_of(nodes[bin], ch[0], ch[1]);
    while (n < 4)
    {
        int best = -1;
        double bestA = -1.0;
        for (int k = 0; k < n; ++k)
            if (ch[k].link >= 0 && half_area(ch[k]) > bestA)
            {
                best = k;
                bestA = half_area(ch[k]);
            }
        if (best < 0)
            break;
        if (ch[best].link >= count)
            return 0;
        opened |= (best + 1) << (4 * (n - 2));
        open_child(nodes, ch, n, best);
    }
    for (int k = 0; k < n; ++k)
        if (ch[k].link >= count)
            return 0;
    return n;
}

// The nodes of a level: [bound[level], level_end). None once links are no
// tree: the count of nodes may then be past the arrays.
__host__ __device__ inline int level_end(const WideCounters& c, int level, int count)
{
    return c.error || c.bound[level + 1] > count ? 0 : c.bound[level + 1];
}

// Takes wide node i: takes consecutive nodes of the next level for the inner
// ones of its children (one atomic).
__host__ __device__ inline void collapse_node(const DevNode* nodes, int count, WideItem* items, WideCounters* c, int i)
{
    const WideItem it = items[i];
    WideChild ch[4];
    int opened;
    const int n = wide_children(nodes, count, it.bin, ch, opened);
    int inner = 0;
    for (int k = 0; k < n; ++k)
        inner += ch[k].link >= 0 ? 1 : 0;
#ifdef __CUDA_ARCH__
    int node = n > 0 ? atomicAdd(&c->nodes, inner) : 0;
#else
    int node = c->nodes;
    c->nodes += inner;
#endif
    if (n == 0 || node + inner > count)
    {
        c->error = 1;
        return;
    }
    const int need = it.need + (n - 1);
#ifdef __CUDA_ARCH__
    atomicMax(&c->maxNeed, need);
#else
    c->maxNeed = need > c->maxNeed ? need : c->maxNeed;
#endif
    items[i].child = node;
    items[i].opened = opened;
    for (int k = 0; k < n; ++k)
        if (ch[k].link >= 0)
            items[node++] = WideItem{ ch[k].link, need, 0, 0 };
}

// Writes wide node i of a tree that collapse_node has taken without an error.
__host__ __device__ inline void write_node(const DevNode* nodes, const WideItem* items, DevNode4* wide, int i)
{
    const WideItem it = items[i];
    WideChild ch[4];
    int n = 2;
    children_of(nodes[it.bin], ch[0], ch[1]);
    for (int o = it.opened; o != 0; o >>= 4)
        open_child(nodes, ch, n, (o & 15) - 1);
    int node = it.child;
    DevNode4 w{};
    float* lox = &w.lox.x;
    float* hix = &w.hix.x;
    float* loy = &w.loy.x;
    float* hiy = &w.hiy.x;
    float* loz = &w.loz.x;
    float* hiz = &w.hiz.x;
    int* link = &w.link.x;
    for (int k = 0; k < n; ++k)
    {
        lox[k] = ch[k].lo[0];
        hix[k] = ch[k].hi[0];
        loy[k] = ch[k].lo[1];
        hiy[k] = ch[k].hi[1];
        loz[k] = ch[k].lo[2];
        hiz[k] = ch[k].hi[2];
        link[k] = ch[k].link >= 0 ? node++ : ch[k].link;
    }
    w.meta.x = n;
    wide[i] = w;
}

// One level of a collapse: takes its nodes, at most `most`, and closes the next.
cudaError_t launch_collapse(const DevNode* nodes, int count, WideItem* items, WideCounters* c, int level, size_t most,
                            int numSMs, cudaStream_t stream);
// The taken nodes, written.
cudaError_t launch_write_nodes(const DevNode* nodes, const WideItem* items, DevNode4* wide, int taken,
                               cudaStream_t stream);

}  // namespace rcx
