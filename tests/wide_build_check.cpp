// Host check of wide_host.cpp against a CUDA runtime whose device is host
// memory: allocations can be made to fail, and a level of nodes is taken one
// by one, with the kernels' own steps. Built with the address sanitizer.

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <utility>
#include <vector>

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

cudaError_t launch_collapse(const DevNode* nodes, int count, WideItem* items, WideCounters* c, int level, size_t, int,
                            cudaStream_t)
{
    const int end = level_end(*c, level, count);
    for (int i = c->bound[level]; i < end; ++i)
        collapse_node(nodes, count, items, c, i);
    c->bound[level + 2] = c->nodes;
    return cudaSuccess;
}

cudaError_t launch_write_nodes(const DevNode* nodes, const WideItem* items, DevNode4* wide, int taken,
                               cudaStream_t)
{
    for (int i = 0; i < taken; ++i)
        write_node(nodes, items, wide, i);
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

// A random binary tree of `count` inner nodes in preorder (leaf codes
// ~(slot << 4 | 1), slots in order), its boxes nested.
std::vector<rcx::DevNode> random_tree(int count, unsigned seed)
{
    std::mt19937 rng(seed);
    std::vector<rcx::DevNode> nodes(static_cast<size_t>(count));
    int next = 0, leaf = 0;
    // inner nodes of the subtree at `node`, its box
    struct Box
    {
        float lo[3], hi[3];
    };
    auto grow = [&](auto&& self, int inner, Box box) -> int {
        const int me = next++;
        const int left = int(rng() % unsigned(inner));  // of the inner - 1 others
        const int n[2] = { left, inner - 1 - left };
        for (int k = 0; k < 2; ++k)
        {
            Box b = box;
            const int axis = int(rng() % 3);
            (k ? b.lo : b.hi)[axis] = b.lo[axis] + (b.hi[axis] - b.lo[axis]) * (0.3f + 0.4f * float(rng() % 1000) / 1000.0f);
            (k ? nodes[size_t(me)].xy1 : nodes[size_t(me)].xy0) = make_float4(b.lo[0], b.hi[0], b.lo[1], b.hi[1]);
            (k ? nodes[size_t(me)].z01.z : nodes[size_t(me)].z01.x) = b.lo[2];
            (k ? nodes[size_t(me)].z01.w : nodes[size_t(me)].z01.y) = b.hi[2];
            int link = ~((leaf << rcx::kLeafCountBits) | 1);
            if (n[k] > 0)
                link = self(self, n[k], b);
            else
                leaf++;
            (k ? nodes[size_t(me)].link.y : nodes[size_t(me)].link.x) = link;
        }
        return me;
    };
    grow(grow, count, Box{ { -1.0f, -1.0f, -1.0f }, { 1.0f, 1.0f, 1.0f } });
    return nodes;
}

int depth_of(const std::vector<rcx::DevNode>& nodes, int link)
{
    if (link < 0)
        return 1;
    return 1 + std::max(depth_of(nodes, nodes[size_t(link)].link.x), depth_of(nodes, nodes[size_t(link)].link.y));
}

// A tracer with a scene of these inner nodes (also the two-level scene's top level).
void scene(rc_tracer& h, std::vector<rcx::DevNode>& nodes, int levels, int instances)
{
    h.sceneReady = true;
    h.numSMs = 4;
    h.innerCount = nodes.size();
    h.rootLink = 0;
    h.bvhDepth = uint64_t(instances > 0 ? 2 * levels : levels);
    h.tlasDepth = uint32_t(instances > 0 ? levels : 0);
    h.dNodes = nodes.data();
    h.nInstances = instances;
    h.tlasRoot = 0;
    h.tlasCount = nodes.size();
    h.dTlas = nodes.data();
    h.instRoots.assign(size_t(instances), 0);
}

void release(rc_tracer& h)
{
    cudaFree(h.dWide);
    cudaFree(h.dWideTlas);
    cudaFree(h.dInstWide);
    CHECK(live.empty());
}

// Leaf slots below a wide node, and the wide nodes (`used`).
void leaves(const rcx::DevNode4* wide, int link, std::vector<int>& out, size_t& used)
{
    if (link < 0)
    {
        out.push_back((~link) >> rcx::kLeafCountBits);
        return;
    }
    used++;
    const int n = wide[link].meta.x;
    CHECK(n >= 2 && n <= 4);
    const int* l = &wide[link].link.x;
    for (int k = 0; k < n; ++k)
        leaves(wide, l[k], out, used);
}

void valid_trees()
{
    for (int count : { 1, 2, 3, 7, 50, 400 })
        for (unsigned seed = 1; seed <= 5; ++seed)
        {
            std::vector<rcx::DevNode> nodes = random_tree(count, seed);
            const int levels = depth_of(nodes, 0);
            if (levels > rcx::kMaxStack)
                continue;
            rc_tracer h;
            scene(h, nodes, levels, 0);
            failAt = 0;
            CHECK(rcx::ensure_wide(&h) == RC_OK);
            if (h.dWide)
            {
                std::vector<int> slots;
                size_t used = 0;
                leaves(h.dWide, h.wideRoot, slots, used);
                CHECK(live[h.dWide] == used * sizeof(rcx::DevNode4));  // no more than the tree's nodes
                std::sort(slots.begin(), slots.end());
                CHECK(int(slots.size()) == count + 1);
                for (int i = 0; i < int(slots.size()); ++i)
                    CHECK(slots[size_t(i)] == i);
            }
            CHECK(live_bytes() == h.deviceBytes);
            release(h);
        }
}

// A wide node opens its child of largest area, compared in 64 bits: of two
// boxes of 16 x 16 x 1 and 16 x 16 x (1 + 2^-23), whose areas round to one
// 32-bit value, the second.
void largest_area()
{
    auto node = [](float h0, int l0, float h1, int l1) {
        rcx::DevNode n{};
        n.xy0 = n.xy1 = make_float4(0.0f, 16.0f, 0.0f, 16.0f);
        n.z01 = make_float4(0.0f, h0, 0.0f, h1);
        n.link = make_int4(l0, l1, 0, 0);
        return n;
    };
    auto leaf = [](int slot) { return ~((slot << rcx::kLeafCountBits) | 1); };
    const float more = 1.0f + 1.0f / 8388608.0f;
    // 0: the large 1 and the box of 2; 1: the box of 3 and a leaf
    const std::vector<rcx::DevNode> nodes{ node(8.0f, 1, more, 2), node(1.0f, 3, 0.5f, leaf(0)),
                                           node(0.1f, leaf(1), 0.1f, leaf(2)), node(0.1f, leaf(3), 0.1f, leaf(4)) };
    rcx::WideChild ch[4];
    int opened;
    CHECK(rcx::wide_children(nodes.data(), 4, 0, ch, opened) == 4);
    bool box3 = false;
    for (const rcx::WideChild& c : ch)
        box3 |= c.link == 3;
    CHECK(box3);  // left as it is: the box of 2 is opened
}

// Links that are no tree: reported, and nothing outside the arrays is read or
// written (the address sanitizer).
void malformed_links()
{
    for (unsigned seed = 1; seed <= 40; ++seed)
    {
        std::mt19937 rng(seed);
        const int count = 2 + int(rng() % 60);
        std::vector<rcx::DevNode> nodes = random_tree(count, seed);
        const int levels = rcx::kMaxStack;
        const size_t at = rng() % nodes.size();
        int& link = (rng() & 1) ? nodes[at].link.x : nodes[at].link.y;
        switch (seed % 4)
        {
        case 0: link = count; break;                // past the nodes
        case 1: link = count + 1000000; break;
        case 2: link = 0; break;                    // a cycle
        default:                                    // every node twice
            for (int i = 0; i + 1 < count; ++i)
                nodes[size_t(i)].link = make_int4(i + 1, i + 1, 0, 0);
        }
        rc_tracer h;
        scene(h, nodes, levels, 0);
        failAt = 0;
        const rc_status s = rcx::ensure_wide(&h);
        CHECK(s == RC_DEVICE_ERROR || (s == RC_OK && !h.dWide));
        if (seed % 4 < 2)
            CHECK(s == RC_DEVICE_ERROR);
        release(h);
    }
    // roots outside the nodes
    for (int root : { 50, 1 << 30 })
    {
        std::vector<rcx::DevNode> nodes = random_tree(50, 1);
        rc_tracer h;
        scene(h, nodes, rcx::kMaxStack, 2);
        h.instRoots[1] = root;
        CHECK(rcx::ensure_wide(&h) == RC_DEVICE_ERROR);
        release(h);
    }
}

// Without memory for a 4-wide tree a scene stays binary: no error, nothing
// left behind, and the next call neither fails nor tries again.
void allocation_failures()
{
    std::vector<rcx::DevNode> nodes = random_tree(400, 1);
    for (int instances : { 0, 3 })
        for (int at = 1; at <= 6; ++at)
        {
            rc_tracer h;
            scene(h, nodes, depth_of(nodes, 0), instances);
            allocations = 0;
            failAt = at;
            failWith = cudaErrorMemoryAllocation;
            CHECK(rcx::ensure_wide(&h) == RC_OK);
            CHECK(h.err.empty());
            if (allocations >= failAt)
                CHECK(instances == 0 ? !h.dWide : !h.wideInstanced);
            CHECK(live_bytes() == h.deviceBytes);
            CHECK(rcx::ensure_wide(&h) == RC_OK);
            release(h);
        }
    // another error is reported
    rc_tracer h;
    scene(h, nodes, depth_of(nodes, 0), 0);
    allocations = 0;
    failAt = 1;
    failWith = cudaErrorUnknown;
    CHECK(rcx::ensure_wide(&h) == RC_CUDA);
    CHECK(live.empty());
}

}  // namespace

int main()
{
    valid_trees();
    largest_area();
    malformed_links();
    allocation_failures();
    if (!failures)
        std::printf("wide build ok\n");
    return failures ? 1 : 0;
}
