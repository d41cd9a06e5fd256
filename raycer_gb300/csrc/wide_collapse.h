// Records and launches of the 4-wide trees' construction: the kernels are in
// wide_build.cu, the host side in wide_host.cpp.
#pragma once

#include <cuda_runtime.h>

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
};

// What a wide node is made from.
struct WideItem
{
    int bin;   // its binary inner node
    int need;  // stack entries pushed above it
};

// One level of a collapse: closes the level above and takes its nodes, at
// most `most` of them.
cudaError_t launch_collapse(const DevNode* nodes, int count, WideItem* items, DevNode4* wide, WideCounters* c,
                            int level, size_t most, int numSMs, cudaStream_t stream);

}  // namespace rcx
