// Ray-casting kernels: generic closest/any-hit queries and the RAY tracer's
// frame (one primary ray per pixel + one shadow ray per hit).
//
// Work distribution: persistent blocks (occupancy x SM count) whose warps
// take 32 rays (an 8x4-pixel tile of a whole frame) at a time from a global
// atomic work counter. An uncounted RAY frame is one kernel: each lane whose
// primary ray hit traces its shadow ray right after its tile. Counted frames
// (and RC_TRACE_FUSED=0) keep two stages: the shadow stage is fed by a queue
// that the primary stage fills with one atomicAdd per warp after a ballot
// over the lanes that hit (warp-aggregated compaction), so shadow warps
// carry no missed pixels.

#include <cfloat>
#include <cmath>

#include "kernels.h"
#include <cstdlib>

#include "monitor.cuh"

#include "traverse.cuh"

namespace rcx
{
namespace
{

constexpr int kBlock = 128;

// Minimum resident blocks per SM the ray kernels are compiled for (register
// budget: 10 blocks x 128 threads -> at most 48 registers, no spills).
#ifndef RC_TRACE_MIN_BLOCKS
#define RC_TRACE_MIN_BLOCKS 10
#endif
// The one-kernel RAY frame (primary + shadow walks) of a single-level scene at
// 7 blocks (it takes 60-64 registers, so 8 are resident): it is bound by issue,
// and on frames of few tiles per warp by the chain of the longest tile; with
// registers to spare the compiler orders the fetches better, which the warps
// of a ninth block (56 registers) do not make up for. 7 / 8 / 9 blocks, 1M
// triangles: 1080p 392 / 394 / 398 us, 640x360 192 / 199 / 203, in reference
// order 836 / 875 / 855 and 719 / 753 / 782; 6 and 5 blocks as 7. Two-level
// frames keep 9.
#ifndef RC_FUSED_MIN_BLOCKS
#define RC_FUSED_MIN_BLOCKS 7
#endif
#ifndef RC_FUSED_INST_MIN_BLOCKS
#define RC_FUSED_INST_MIN_BLOCKS 9
#endif
#ifndef RC_TRACE_TILES
#define RC_TRACE_TILES 1
#endif
constexpr int kWarpsPerBlock = kBlock / 32;

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned warp_fetch(unsigned* head, unsigned amount)
{
    unsigned base = 0;
    if (lane_id() == 0)
        base = atomicAdd(head, amount);
    return __shfl_sync(0xffffffffu, base, 0);
}

__device__ __forceinline__ void flush_counts(DevControl* ctl, int stage, unsigned long long rays, const TravCount& c,
                                             int err)
{
    unsigned long long n = c.nodes, t = c.tris;
    for (int o = 16; o > 0; o >>= 1)
    {
        rays += __shfl_down_sync(0xffffffffu, rays, o);
        n += __shfl_down_sync(0xffffffffu, n, o);
        t += __shfl_down_sync(0xffffffffu, t, o);
    }
    if (lane_id() == 0)
    {
        atomicAdd(&ctl->stats[3 * stage + 0], rays);
        if (n)
            atomicAdd(&ctl->stats[3 * stage + 1], n);
        if (t)
            atomicAdd(&ctl->stats[3 * stage + 2], t);
    }
    if (err)
        atomicOr(&ctl->error, 1);
}

template <bool C, typename A, typename B>
struct Choose
{
    using type = A;
};
template <typename A, typename B>
struct Choose<false, A, B>
{
    using type = B;
};

__device__ __forceinline__ int caller_index(const DevScene& sc, int slot)
{
    return __float_as_int(__ldg(&sc.tris[slot].c.z));
}

// Large casts are launched twice, straight (k_cast) and in phases
// (k_cast_phased), and the samples of k_cast_samples decide on the device which
// of the two does the work: `run` is the answer a kernel waits for, or kAnyRays.
enum CastRun
{
    kApart = 0,
    kTogether = 1,
    kAnyRays = 2
};
constexpr int kCastSamples = 32;

__device__ __forceinline__ bool cast_runs(const DevControl* ctl, int run)
{
    return run == kAnyRays ||
           run == (*reinterpret_cast<const volatile unsigned*>(&ctl->head[1]) * 2u >= unsigned(kCastSamples) ? kTogether
                                                                                                          : kApart);
}

template <bool ANY, int ORDER, bool COUNT, bool SL>
__global__ void __launch_bounds__(kBlock, RC_TRACE_MIN_BLOCKS) k_cast(DevScene sc, const rc_ray* __restrict__ rays, int n,
                                                 rc_hit* __restrict__ hits, DevControl* ctl, int run)
{
    if (!cast_runs(ctl, run))
        return;
    TravCount cnt{ 0, 0 };
    int err = 0;
    unsigned long long done = 0;
    while (true)
    {
        unsigned base = warp_fetch(&ctl->head[0], 32u);
        if (base >= unsigned(n))
            break;
        int i = int(base + lane_id());
        if (i < n)
        {
            const float4* rp = reinterpret_cast<const float4*>(rays + i);
            float4 r0 = __ldg(rp);
            float4 r1 = __ldg(rp + 1);
            RayF ray = make_ray(v3(r0.x, r0.y, r0.z), v3(r1.x, r1.y, r1.z), r0.w, r1.w);
            HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
            // SL: the reference order of a single-level scene on the rope records
            bool found = SL ? traverse_stackless<ANY>(sc, ray, h, -1)
                            : traverse_scene<ANY, ORDER, COUNT>(sc, ray, h, cnt, err, -1, -1);
            int4 out;
            // two-level scenes: the flattened index (instance's first + mesh-local)
            out.x = found ? caller_index(sc, h.slot) + (h.inst >= 0 ? __ldg(&sc.instances[h.inst].primBase) : 0) : -1;
            out.y = __float_as_int(found ? h.t : -1.0f);
            out.z = __float_as_int(found ? h.u : 0.0f);
            out.w = __float_as_int(found ? h.v : 0.0f);
            reinterpret_cast<int4*>(hits)[i] = out;
            done++;
        }
    }
    flush_counts(ctl, 0, done, cnt, err);
}

__device__ __forceinline__ RayF primary_ray(const DevCamera& cam, const rc_ray* __restrict__ rays, uint64_t pixel,
                                            int64_t local, int64_t width)
{
    if (rays)
    {
        const float4* rp = reinterpret_cast<const float4*>(rays + local);
        float4 r0 = __ldg(rp);
        float4 r1 = __ldg(rp + 1);
        return make_ray(v3(r0.x, r0.y, r0.z), v3(r1.x, r1.y, r1.z), r0.w, r1.w);
    }
    float px = float(pixel % uint64_t(width));
    float py = float(pixel / uint64_t(width));
    V3 d = camera_dir(cam, px, py);
    return make_ray(v3(cam.pos[0], cam.pos[1], cam.pos[2]), d, 0.0f, FLT_MAX);
}

// The shadow ray of a primary hit, traced where the hit was found: the
// arithmetic of stage 2 below (origin = o + t d, then + L * rayStartOffset;
// the hit's own triangle, of its instance, skipped). Completes the record:
// occluder and flags.
// SOCT >= 0: the light's direction has the signs of octant SOCT (the host
// checked that its inverse is finite), and the walk's box tests use them
// (slab_oct: the same decisions, six FMNMX fewer per box).
template <bool INST, bool SL, int SOCT = -1>
__device__ __forceinline__ void shadow_of(const DevScene& sc, const RayF& ray, const HitF& h, float3 L,
                                          float rayStartOffset, int4& o, TravCount& cnt, int& err)
{
    const V3 dl = v3(L.x, L.y, L.z);
    const RayF sr = make_ray(vfma(dl, rayStartOffset, vfma(ray.d, h.t, ray.o)), dl, 0.0f, FLT_MAX);
    HitF s{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
    bool occ;
    if (INST)
        occ = traverse_instanced<true, false>(sc, sr, s, cnt, err, h.slot, h.inst);
    else if (SL)
        occ = traverse_stackless<true>(sc, sr, s, h.slot);
    else
        occ = traverse<true, ORDER_REF, false, SOCT>(sc, sr, s, cnt, err, h.slot);
    o.z = occ ? caller_index(sc, s.slot) + (INST ? __ldg(&sc.instances[s.inst].primBase) : 0) : -1;
    o.w = 1 | 2 | (occ ? 4 : 0);
}

// Stage 1 of the RAY frame: closest hit of every pixel's primary ray.
// Camera rays (and caller rays, one per pixel of a whole frame) are
// walked in 8x4-pixel tiles, one tile per warp fetch, so a warp's rays are
// spatially coherent.
// PACKET: the warp traverses its 32 rays together (traverse_packet); the
// counted frame keeps one traversal per lane, whose node and triangle counts
// are the algorithm's. INST: a two-level scene (traverse_instanced; the
// record's prim is the flattened index, instance's first + mesh-local, and
// while a shadow ray is to follow its occluder field holds the hit's
// instance, for the shadow ray to skip the hit triangle of that instance).
// FUSED (uncounted frames with a light): each lane whose ray hit traces its
// shadow ray right after the tile's primary rays, with the shadow kernel's
// arithmetic (stage 2 below; SL: the stackless walk), and the pixel's record
// is written once, complete; no queue. The shadow rays of a tile whose
// pixels all hit (or all miss) keep the warp full (or cost nothing); only
// tiles on a silhouette leave lanes idle. With the caller's rays in host
// memory the shadow work then overlaps the ray reads over the host link.
template <int ORDER, bool COUNT, bool PACKET, bool INST, bool FUSED = false, bool SL = false, int SOCT = -1>
__global__ void __launch_bounds__(kBlock, !FUSED ? RC_TRACE_MIN_BLOCKS
                                          : INST ? RC_FUSED_INST_MIN_BLOCKS
                                                 : RC_FUSED_MIN_BLOCKS)
    k_raycast_primary(DevScene sc, DevCamera cam, const rc_ray* __restrict__ rays,
                                                            uint64_t pixelStart, int64_t count, int64_t width,
                                                            FilmTiles tiles, int castShadow,
                                                            rc_cast_pixel* __restrict__ out, int* __restrict__ queue,
                                                            DevControl* ctl, float3 L, float rayStartOffset,
                                                            float4* __restrict__ origins)
{
    static_assert(!(FUSED && COUNT), "counted frames keep the two stages");
    TravCount cnt1{ 0, 0 };  // FUSED: the shadow rays' counts
    unsigned long long done1 = 0;
    __shared__ PacketEntry wstack[PACKET ? kWarpsPerBlock : 1][PACKET ? kMaxStack : 1];
    TravCount cnt{ 0, 0 };
    int err = 0;
    unsigned long long done = 0;
    const int64_t items = tile_items(tiles, count);
    if (is_watch_warp(sc.monitor, sc.budgetNs))
    {
        watch_queue(sc.monitor, sc.budgetNs, ctl, &ctl->head[0], static_cast<unsigned long long>(items),
                    FUSED ? kPublishEstimate : kPublishNone, static_cast<unsigned long long>(count), nullptr, tiles);
        return;
    }
    while (true)
    {
        unsigned base = warp_fetch(&ctl->head[0], 32u);
        if (int64_t(base) >= items)
            break;
        int64_t i;
        const bool valid = tile_pixel(tiles, count, int64_t(base) + lane_id(), i);
        bool hitAny = false;
        int hitSlot = -1;
        float4 sorg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // shadow-ray origin (+ instance) for `origins`
        if (PACKET)
        {
            // all lanes together, the ray of an invalid lane unused
            RayF ray = primary_ray(cam, rays, valid ? pixelStart + uint64_t(i) : pixelStart, valid ? i : 0, width);
            HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
            bool found = traverse_packet<ORDER>(sc, ray, h, err, -1, valid, wstack[threadIdx.x >> 5]);
            // the one-kernel and two-stage records are built apart: one shared
            // branch measured 1 % slower on the one-kernel frame
            if (FUSED)
            {
                int4 o;
                o.x = found ? caller_index(sc, h.slot) : -1;
                o.y = __float_as_int(found ? h.t : -1.0f);
                o.z = -1;
                o.w = found ? 1 : 0;
                if (valid && found)
                    shadow_of<false, SL, SOCT>(sc, ray, h, L, rayStartOffset, o, cnt1, err);
                if (valid)
                {
                    reinterpret_cast<int4*>(out)[i] = o;
                    done++;
                    done1 += found ? 1 : 0;
                }
            }
            else if (valid)
            {
                int4 o;
                o.x = found ? caller_index(sc, h.slot) : -1;
                o.y = __float_as_int(found ? h.t : -1.0f);
                o.z = -1;
                o.w = found ? 1 : 0;
                reinterpret_cast<int4*>(out)[i] = o;
                hitAny = found && castShadow;
                hitSlot = h.slot;
                if (origins && hitAny)
                {
                    // the shadow kernel's own arithmetic (ip = o + t d, then + L * offset)
                    const V3 dl = v3(L.x, L.y, L.z);
                    const V3 so = vfma(dl, rayStartOffset, vfma(ray.d, h.t, ray.o));
                    sorg = make_float4(so.x, so.y, so.z, __int_as_float(-1));
                }
                done++;
            }
        }
        else if (valid)
        {
            RayF ray = primary_ray(cam, rays, pixelStart + uint64_t(i), i, width);
            HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
            bool found;
            if (INST)
                found = traverse_instanced<false, COUNT>(sc, ray, h, cnt, err, -1, -1);
            else
                found = traverse<false, ORDER, COUNT>(sc, ray, h, cnt, err);
            int4 o;
            o.x = found ? caller_index(sc, h.slot) + (INST ? __ldg(&sc.instances[h.inst].primBase) : 0) : -1;
            o.y = __float_as_int(found ? h.t : -1.0f);
            o.z = INST && found && castShadow && !FUSED ? h.inst : -1;
            o.w = found ? 1 : 0;
            if (FUSED)
            {
                if (found)
                {
                    shadow_of<INST, SL, INST ? -1 : SOCT>(sc, ray, h, L, rayStartOffset, o, cnt1, err);
                    done1++;
                }
            }
            else if (origins && found && castShadow)
            {
                const V3 dl = v3(L.x, L.y, L.z);
                const V3 so = vfma(dl, rayStartOffset, vfma(ray.d, h.t, ray.o));
                sorg = make_float4(so.x, so.y, so.z, __int_as_float(INST ? h.inst : -1));
            }
            reinterpret_cast<int4*>(out)[i] = o;
            hitAny = found && castShadow && !FUSED;
            hitSlot = h.slot;
            done++;
        }
        // Warp-aggregated compaction of the hit pixels into the shadow queue.
        unsigned mask = FUSED ? 0u : __ballot_sync(0xffffffffu, hitAny);
        if (mask)
        {
            unsigned qbase = 0;
            if (lane_id() == 0)
                qbase = atomicAdd(&ctl->head[1], unsigned(__popc(mask)));
            qbase = __shfl_sync(0xffffffffu, qbase, 0);
            if (hitAny)
            {
                const unsigned qi = qbase + __popc(mask & ((1u << lane_id()) - 1u));
                reinterpret_cast<int2*>(queue)[qi] = make_int2(int(i), hitSlot);
                if (origins)
                    origins[qi] = sorg;
            }
        }
    }
    flush_counts(ctl, 0, done, cnt, err);
    if (FUSED)
        flush_counts(ctl, 1, done1, cnt1, 0);
}

// Stage 2: one any-hit shadow ray toward the light per queued pixel
// (Raytracer::calculateShadowAmount, Raytracer.cpp:497-522 /
// lighting.cl:28-48): origin = hit position + dirToLight * rayStartOffset;
// the primary hit's own triangle is skipped (see traverse.cuh).
template <bool COUNT, bool INST, bool SL>
__global__ void __launch_bounds__(kBlock, RC_TRACE_MIN_BLOCKS) k_raycast_shadow(DevScene sc, DevCamera cam, const rc_ray* __restrict__ rays,
                                                           uint64_t pixelStart, int64_t width, float3 L,
                                                           float rayStartOffset, rc_cast_pixel* __restrict__ out,
                                                           const int* __restrict__ queue, DevControl* ctl,
                                                           const float4* __restrict__ origins)
{
    TravCount cnt{ 0, 0 };
    int err = 0;
    unsigned long long done = 0;
    const unsigned total = *reinterpret_cast<volatile unsigned*>(&ctl->head[1]);
    while (true)
    {
        unsigned base = warp_fetch(&ctl->head[2], 32u);
        if (base >= total)
            break;
        unsigned q = base + lane_id();
        if (q < total)
        {
            int2 e = reinterpret_cast<const int2*>(queue)[q];
            int i = e.x;
            V3 dl = v3(L.x, L.y, L.z);
            RayF sr;
            int skipInst = -1;
            if (origins)
            {
                // stored by the primary kernel with the arithmetic below
                const float4 so = origins[q];
                sr = make_ray(v3(so.x, so.y, so.z), dl, 0.0f, FLT_MAX);
                skipInst = __float_as_int(so.w);
            }
            else
            {
                RayF pr = primary_ray(cam, rays, pixelStart + uint64_t(i), i, width);
                float t = out[i].t;
                // ip = origin + t * direction (intersections.cl:85)
                V3 ip = vfma(pr.d, t, pr.o);
                sr = make_ray(vfma(dl, rayStartOffset, ip), dl, 0.0f, FLT_MAX);
                if (INST)
                    skipInst = out[i].occluder;  // the primary stage left the hit's instance there
            }
            HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
            bool occ;
            if (INST)
                occ = traverse_instanced<true, COUNT>(sc, sr, h, cnt, err, e.y, skipInst);
            else if (SL)
                occ = traverse_stackless<true>(sc, sr, h, e.y);  // the same first occluder, no stack
            else
                occ = traverse<true, ORDER_REF, COUNT>(sc, sr, h, cnt, err, e.y);
            out[i].occluder = occ ? caller_index(sc, h.slot) + (INST ? __ldg(&sc.instances[h.inst].primBase) : 0) : -1;
            out[i].flags = 1 | 2 | (occ ? 4 : 0);
            done++;
        }
    }
    flush_counts(ctl, 1, done, cnt, err);
}

// Large batches of queries in warp-wide phases (as the path tracer's bounce
// kernel): each turn the warp takes the node step or the leaf step that more
// lanes wait for, and once kCastLanes walks have ended, those lanes write
// their hits and take new rays. Nearest-first closest hits walk the 4-wide
// tree; a hit that lies before its own leaf's entry may have been decided by
// the order of the walk (see traverse_group) and is walked again alone, and so
// is a ray whose walk ends undecided.
// Reference-order and any-hit queries take the binary tree's boxes and
// triangles in the reference's order.
//
// Device time of 4M / 1M random rays in 1M triangles, one ray per lane to its
// end (k_cast) -> phases: closest 2,043 -> 1,272 /
// 695 -> 520 us, any hit 2,176 -> 1,278 / 766 -> 591. Hits written
// and rays taken at 8 / 16 / 24 finished lanes: 1,201 / 1,198 / 1,231 us; 8, 9
// and 10 blocks per SM: 1,198 / 1,223 / 1,347 (any hit 1,274 / 1,333 / 1,414).
constexpr int kCastLanes = 16;

__device__ __forceinline__ RayF load_ray(const rc_ray* __restrict__ r)
{
    const float4* p = reinterpret_cast<const float4*>(r);
    const float4 a = __ldg(p);
    const float4 b = __ldg(p + 1);
    return make_ray(v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), a.w, b.w);
}

__device__ __forceinline__ void write_hit(const DevScene& sc, const HitF& h, rc_hit* out)
{
    const bool found = h.slot >= 0;
    *reinterpret_cast<int4*>(out) =
        make_int4(found ? caller_index(sc, h.slot) : -1, __float_as_int(found ? h.t : -1.0f),
                  __float_as_int(found ? h.u : 0.0f), __float_as_int(found ? h.v : 0.0f));
}

// How many of 32 samples of 32 consecutive rays, spread over the batch, would
// walk together: directions within `spread` of the first one's (of its largest
// component), origins within a 32nd of the scene. Camera rays in the order of a
// frame do. One block.
__global__ void __launch_bounds__(kCastSamples * 32) k_cast_samples(DevScene sc, const rc_ray* __restrict__ rays, int n,
                                                                    float spread, DevControl* ctl)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int64_t last = n / 32 - 1;  // of the batch's whole groups of 32
    const int64_t group = last * int64_t(threadIdx.x >> 5) / (kCastSamples - 1);
    const RayF r = load_ray(rays + group * 32 + lane_id());
    float4 a, b, c;
    int4 l;
    load_node(sc.nodes, sc.rootLink, a, b, c, l);
    const float extent = fmaxf(fmaxf(fmaxf(a.y, b.y) - fminf(a.x, b.x), fmaxf(a.w, b.w) - fminf(a.z, b.z)),
                               fmaxf(c.y, c.w) - fminf(c.x, c.z));
    const V3 o = v3(__shfl_sync(kAll, r.o.x, 0), __shfl_sync(kAll, r.o.y, 0), __shfl_sync(kAll, r.o.z, 0));
    const V3 d = v3(__shfl_sync(kAll, r.d.x, 0), __shfl_sync(kAll, r.d.y, 0), __shfl_sync(kAll, r.d.z, 0));
    const float away = fmaxf(fmaxf(fabsf(r.o.x - o.x), fabsf(r.o.y - o.y)), fabsf(r.o.z - o.z));
    const float turn = fmaxf(fmaxf(fabsf(r.d.x - d.x), fabsf(r.d.y - d.y)), fabsf(r.d.z - d.z));
    const float size = fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    if (__all_sync(kAll, away <= extent * (1.0f / 32.0f) && turn <= spread * size) && lane_id() == 0)
        atomicAdd(&ctl->head[1], 1u);
}

template <bool ANY, int ORDER>
__global__ void __launch_bounds__(kBlock, 8) k_cast_phased(DevScene sc, const rc_ray* __restrict__ rays, int n,
                                                           rc_hit* __restrict__ hits, DevControl* ctl, int run)
{
    if (!cast_runs(ctl, run))
        return;
    constexpr unsigned kAll = 0xffffffffu;
    constexpr bool WIDE = !ANY && ORDER == ORDER_NEAREST;
    constexpr int kNear = WIDE ? 12 : 16;  // stack entries in shared memory
    using Entry = typename Choose<WIDE, int2, int>::type;
    using Walk = typename Choose<WIDE, CastWalk, RefWalk>::type;
    __shared__ Entry nearEntries[kNear][kBlock];
    Entry farEntries[kMaxStack - kNear];
    SharedStack<kNear, kBlock, kMaxStack, Entry> stack{ &nearEntries[0][threadIdx.x], farEntries };
    // rays to walk again alone: out of the loop, which the call would make spill
    __shared__ int again[kWarpsPerBlock][WIDE ? 64 : 1];
    int* list = again[threadIdx.x >> 5];
    const unsigned below = (1u << lane_id()) - 1u;
    int listed = 0;        // warp-uniform
    unsigned done = 0;     // warp-uniform
    bool drained = false;  // warp-uniform
    int err = 0;
    while (true)
    {
        int i = 0;  // this lane's ray
        RayF ray = make_ray(v3(0.0f, 0.0f, 0.0f), v3(1.0f, 1.0f, 1.0f), 0.0f, FLT_MAX);
        HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
        Walk w{};
        w.cur = kWalkNone;
        while (true)
        {
            const unsigned atNode = __ballot_sync(kAll, w.cur >= 0);
            const unsigned atLeaf = __ballot_sync(kAll, w.cur < 0 && w.cur > kWalkNone);
            const bool take = !drained && listed < 32;
            const unsigned waiting = __ballot_sync(kAll, w.cur == kWalkDone || (w.cur == kWalkNone && take));
            if (waiting && ((atNode | atLeaf) == 0u || __popc(waiting) >= kCastLanes))
            {
                done += unsigned(__popc(__ballot_sync(kAll, w.cur == kWalkDone)));
                if constexpr (WIDE)
                {
                    // no hit: 0 within FLT_MAX; undecided: a NaN
                    const bool odd = w.cur == kWalkDone && !(w.hitEntry <= h.t);
                    const unsigned m = __ballot_sync(kAll, odd);
                    if (odd)
                        list[listed + __popc(m & below)] = i;
                    listed += __popc(m);
                }
                if (w.cur == kWalkDone)
                {
                    write_hit(sc, h, hits + i);
                    w.cur = kWalkNone;
                }
                // decided after this turn's rays are listed: the 31 of a list
                // with room and the 32 that may be in flight fit its 64 entries
                const unsigned idle = __ballot_sync(kAll, w.cur == kWalkNone);
                if (!drained && listed < 32)
                {
                    const unsigned base = warp_fetch(&ctl->head[0], unsigned(__popc(idle)));
                    drained = base + unsigned(__popc(idle)) >= unsigned(n);
                    const unsigned q = base + unsigned(__popc(idle & below));
                    if (((idle >> lane_id()) & 1u) && q < unsigned(n))
                    {
                        i = int(q);
                        ray = load_ray(rays + i);
                        h = HitF{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
                        w = Walk{};
                        w.cur = WIDE ? sc.wideRoot : sc.rootLink;
                    }
                }
                continue;
            }
            if ((atNode | atLeaf) == 0u)
                break;
            if (__popc(atLeaf) > __popc(atNode))
            {
                if (w.cur < 0 && w.cur > kWalkNone)
                {
                    if constexpr (WIDE)
                        wide_leaf_step(sc.tris, ray, h, w, stack, -1);
                    else
                        ref_leaf_step<ANY>(sc.tris, ray, h, w, stack, -1);
                }
            }
            else if (w.cur >= 0)
            {
                if constexpr (WIDE)
                    wide_node_step(sc.wide, ray, h, w, stack, err);
                else
                    ref_node_step(sc.nodes, ray, w, stack);
            }
        }
        if (WIDE)
        {
            __syncwarp();
            for (int k = int(lane_id()); k < listed; k += 32)
            {
                const int r = list[k];
                const RayF alone = load_ray(rays + r);
                HitF a;
                traverse_alone<ORDER_NEAREST>(sc, alone, a, -1);
                write_hit(sc, a, hits + r);
            }
            __syncwarp();
            listed = 0;
        }
        if (drained)
            break;
    }
    flush_counts(ctl, 0, lane_id() == 0 ? done : 0u, TravCount{ 0, 0 }, err);
}

// The same queries and frames with a group of G lanes per ray (traverse_group),
// for calls with few rays; 32 / G rays per warp fetch. What bounds them is the
// rounds of dependent fetches of the longest ray, about a twentieth of its
// node count. 8 blocks of 16 KB of stacks leave the SM half its L1. 777 random
// rays in 1M triangles 131 -> 26 us, 100,000 215 -> 170 us; RAY frames of 260k
// triangles at 160x90 226 -> 58 us, at 320x180 199 -> 101 us, in the
// reference's order 791 -> 60 and 482 -> 124 us.
template <bool ANY, int ORDER>
__global__ void __launch_bounds__(kBlock, 8) k_cast_group(DevScene sc, const rc_ray* __restrict__ rays, int n,
                                                       rc_hit* __restrict__ hits, DevControl* ctl, unsigned G,
                                                       int reserve)
{
    __shared__ int2 stacks[kWarpsPerBlock][kGroupEntries];
    const unsigned take = 32u / G;
    const unsigned group = lane_id() / G;
    const int capacity = kGroupEntries / int(take);
    int2* stack = stacks[threadIdx.x >> 5] + int(group) * capacity;
    unsigned long long done = 0;
    while (true)
    {
        const unsigned base = warp_fetch(&ctl->head[0], take);
        if (base >= unsigned(n))
            break;
        const bool active = base + group < unsigned(n);
        const int i = active ? int(base + group) : int(base);
        const RayF ray = load_ray(rays + i);
        HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
        traverse_group<ANY, ORDER>(sc, ray, h, -1, active, G, stack, capacity, reserve);
        if (active && lane_id() % G == 0)
        {
            write_hit(sc, h, hits + i);
            done++;
        }
    }
    flush_counts(ctl, 0, done, TravCount{ 0, 0 }, 0);
}

// The one-kernel RAY frame (primary ray, then the hit's shadow ray).
template <int ORDER>
__global__ void __launch_bounds__(kBlock, 8) k_raycast_group(DevScene sc, DevCamera cam, const rc_ray* __restrict__ rays,
                                                          uint64_t pixelStart, int64_t count, int64_t width,
                                                          FilmTiles tiles, int castShadow,
                                                          rc_cast_pixel* __restrict__ out, DevControl* ctl, float3 L,
                                                          float rayStartOffset, unsigned G, int reserve)
{
    __shared__ int2 stacks[kWarpsPerBlock][kGroupEntries];
    const unsigned take = 32u / G;
    const unsigned group = lane_id() / G;
    const int capacity = kGroupEntries / int(take);
    int2* stack = stacks[threadIdx.x >> 5] + int(group) * capacity;
    unsigned long long done = 0, done1 = 0;
    const int64_t items = tile_items(tiles, count);
    if (is_watch_warp(sc.monitor, sc.budgetNs))
    {
        watch_queue(sc.monitor, sc.budgetNs, ctl, &ctl->head[0], static_cast<unsigned long long>(items),
                    kPublishEstimate, static_cast<unsigned long long>(count), nullptr, tiles);
        return;
    }
    while (true)
    {
        const unsigned base = warp_fetch(&ctl->head[0], take);
        if (int64_t(base) >= items)
            break;
        int64_t i = 0;
        const bool valid = int64_t(base) + group < items && tile_pixel(tiles, count, int64_t(base) + group, i);
        const RayF ray = primary_ray(cam, rays, valid ? pixelStart + uint64_t(i) : pixelStart, valid ? i : 0, width);
        HitF h{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
        const bool found = traverse_group<false, ORDER>(sc, ray, h, -1, valid, G, stack, capacity, reserve);
        int4 o;
        o.x = found ? caller_index(sc, h.slot) : -1;
        o.y = __float_as_int(found ? h.t : -1.0f);
        o.z = -1;
        o.w = found ? 1 : 0;
        if (castShadow)
        {
            // shadow_of's ray
            const V3 dl = v3(L.x, L.y, L.z);
            const RayF sr = make_ray(vfma(dl, rayStartOffset, vfma(ray.d, h.t, ray.o)), dl, 0.0f, FLT_MAX);
            HitF s{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
            const bool occ = traverse_group<true, ORDER_REF>(sc, sr, s, h.slot, valid && found, G, stack, capacity, reserve);
            if (found)
            {
                o.z = occ ? caller_index(sc, s.slot) : -1;
                o.w = 1 | 2 | (occ ? 4 : 0);
            }
        }
        if (valid && lane_id() % G == 0)
        {
            reinterpret_cast<int4*>(out)[i] = o;
            done++;
            done1 += found && castShadow ? 1 : 0;
        }
    }
    flush_counts(ctl, 0, done, TravCount{ 0, 0 }, 0);
    flush_counts(ctl, 1, done1, TravCount{ 0, 0 }, 0);
}

// Persistent grid of a ray kernel: resident blocks per SM (cached per
// device) x the launching handle's SMs.
template <typename K>
int persistent_blocks(K kernel, int numSMs, OccupancyCache& cache)
{
    return blocks_per_sm(kernel, kBlock, 0, cache) * numSMs;
}

// Whether a group of G lanes has the stack for the scene's tree; a deeper tree
// is walked one ray per lane.
bool group_fits(const DevScene& sc, unsigned G) { return int(G) * kGroupEntries / 32 >= sc.depth + 2 * int(G); }

// Lanes per ray of an uncounted cast of n rays on a single-level scene, or 0
// for one ray per lane. Each larger group shortens a ray's chain of fetches but
// gives the warp fewer rays, so a group wins where a call is bound by latency,
// which grows with the scene: n x G may be `most` lanes for groups of 32, 16
// and 8, and `most4` for groups of 4. The lines lie where random rays and rays
// of a frame from above, whichever is earlier, take as long one ray per lane.
// Device time with a group of 32 / 16 / 8 / 4 / none, nearest-first:
//   1,482 triangles  10,000 random   34 /  27 /  26 /  30 /  49 us
//                    10,000 frame    37 /  26 /  22 /  21 /  27
//                    40,000 frame     - /   - /  37 /  27 /  26
//   8,930            40,000 random    - /   - /  51 /  45 /  57
//                    80,000 frame     - /   - /  66 /  45 /  42
//   1M               20,000 random   68 /  53 /  47 /  57 /  76
//                    80,000 random    - /   - / 105 / 102 /  97
//                   120,000 frame     - /   - / 148 / 112 / 113
// any hit:
//   8,930            40,000 random    - /   - /  54 /  57 /  64
//   1M               40,000 random    - /  86 /  89 / 103 /  88
//                    40,000 frame     - /  79 /  72 /  96 / 119
// reference order:
//   8,930            80,000 frame     - /   - /  61 /  44 /  46
//   70,668          160,000 frame     - /   - /   - /  95 / 117
//                   148,200 strip     - /   - /   - /  93 /  84
//   1M              311,000 random    - /   - /   - / 402 / 499
template <bool ANY, int ORDER>
unsigned cast_group_lanes(const DevScene& sc, int64_t n, int blocks)
{
    const int64_t lanes = int64_t(blocks) * kBlock;
    const int bits = scene_bits(sc);
    int64_t most, most4;
    if (bits < 13)
    {
        most = lanes / 2;
        most4 = bits < 10 ? lanes * 2 / 3 : lanes;
    }
    else if (ANY)
    {
        most = lanes * 2;
        most4 = 0;
    }
    else if (ORDER == ORDER_NEAREST)
    {
        most = lanes;
        most4 = lanes * 7 / 4;
    }
    else
    {
        most = lanes * 2;
        most4 = bits < 16 ? lanes * 2 : bits < 17 ? lanes * 3 : lanes * 8;
    }
    for (unsigned G = 32u; G >= 4u; G /= 2u)
        if (n * int64_t(G) <= (G == 4u ? most4 : most))
            return group_fits(sc, G) ? G : 0u;
    return 0u;
}

// The same for a frame of n rays. A tile's neighbouring rays share their
// fetches in a full warp, so a frame gains by groups only while it is bound by
// the latency of one warp's walk, which grows with the scene, and a group's
// time grows with the rays that hit. The line is where frames whose rays all
// hit (a terrain seen from above or in a wide strip) take as long either way;
// it is lanes x (6 log2(triangles) - 39) / 40 rays x lanes. Groups above 4 only
// within one ray per group at a time. Whole frames from above, device time with
// a group of 32 / 16 / 8 / 4 / none:
//   1,482 triangles, 160x90    74 /  45 /  36 /  32 /  34 us
//                    320x180    - /   - /  73 /  45 /  33
//   8,930            120x68    56 /  39 /  37 /  34 /  57
//                    240x135    - /   - /  57 /  41 /  52
//                    320x180    - /   - /   - /  56 /  49
//   34,776           160x90    95 /  58 /  46 /  45 /  87
//                    320x180    - /   - /  97 /  70 /  76
//                    400x225    - /   - /   - /  92 /  74
//   1M               160x90   113 /  70 /  59 /  68 / 278
//                    400x225    - /   - / 184 / 141 / 228
//                    520x290    - /   - /   - / 194 / 207
// A strip of 603x150 pixels: 8,930 triangles 79 / 50 (4 / none), 34,776 94 / 63,
// 260,610 121 / 105, 1M 142 / 174.
unsigned frame_group_lanes(const DevScene& sc, int64_t n, int blocks)
{
    const int64_t lanes = int64_t(blocks) * kBlock;
    const int64_t most = lanes * (6 * scene_bits(sc) - 39) / 40;
    for (unsigned G = 32u; G >= 4u; G /= 2u)
        if (n * int64_t(G) <= (G == 4u ? most : std::min(most, lanes)))
            return group_fits(sc, G) ? G : 0u;
    return 0u;
}

template <bool ANY, int ORDER>
cudaError_t cast_phased(const LaunchInfo& li, const DevScene& sc, const rc_ray* rays, int64_t n, rc_hit* hits,
                        DevControl* ctl, int run = kAnyRays)
{
    auto k = k_cast_phased<ANY, ORDER>;
    static OccupancyCache occ;
    k<<<persistent_blocks(k, li.numSMs, occ), kBlock, 0, li.stream>>>(sc, rays, int(n), hits, ctl, run);
    return cudaGetLastError();
}

template <bool ANY, int ORDER>
cudaError_t cast_group(const LaunchInfo& li, const DevScene& sc, const rc_ray* rays, int64_t n, rc_hit* hits,
                       DevControl* ctl, bool& taken)
{
    auto k = k_cast_group<ANY, ORDER>;
    static OccupancyCache occ;
    const int blocks = persistent_blocks(k, li.numSMs, occ);
    const unsigned G = cast_group_lanes<ANY, ORDER>(sc, n, blocks);
    taken = G != 0u;
    if (!taken)
        return cudaSuccess;
    k<<<blocks, kBlock, 0, li.stream>>>(sc, rays, int(n), hits, ctl, G, sc.depth);
    return cudaGetLastError();
}

template <bool ANY, int ORDER, bool COUNT, bool SL = false>
cudaError_t cast_t(const LaunchInfo& li, const DevScene& sc, const rc_ray* rays, int64_t n, rc_hit* hits,
                   DevControl* ctl, int run = kAnyRays)
{
    auto k = k_cast<ANY, ORDER, COUNT, SL>;
    static OccupancyCache occ;
    k<<<persistent_blocks(k, li.numSMs, occ), kBlock, 0, li.stream>>>(sc, rays, int(n), hits, ctl, run);
    return cudaGetLastError();
}

// A large cast: straight where its rays walk together, else in phases. In
// phases warps lose the coherence that camera rays have, and random rays gain
// lanes: straight -> phases, 4M rays, 8,930 triangles: a frame's rays 240 ->
// 357 us (nearest-first), 214 -> 305 (any hit), 305 -> 393 (reference order),
// random rays 891 -> 709, 853 -> 616, 2,044 -> 1,016; 1M triangles: 667 -> 885,
// 628 -> 761, 1,160 -> 1,203, and 1,436 -> 1,045, 1,322 -> 901, 4,516 -> 2,086.
// The spreads are about those of 32 pixels of a row at the sizes where a frame's
// rays take as long either way (400k-600k pixels; 1M in reference order).
template <bool ANY, int ORDER>
cudaError_t cast_large(const LaunchInfo& li, const DevScene& sc, const rc_ray* rays, int64_t n, rc_hit* hits,
                       DevControl* ctl)
{
    if (sc.rootLink < 0)
        return cast_phased<ANY, ORDER>(li, sc, rays, n, hits, ctl);
    constexpr float spread = !ANY && ORDER == ORDER_REF ? 1.0f / 40.0f : 1.0f / 24.0f;
    k_cast_samples<<<1, kCastSamples * 32, 0, li.stream>>>(sc, rays, int(n), spread, ctl);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cast_t<ANY, ORDER, false>(li, sc, rays, n, hits, ctl, kTogether);
    return e == cudaSuccess ? cast_phased<ANY, ORDER>(li, sc, rays, n, hits, ctl, kApart) : e;
}

// Warp-wide traversal of the primary rays of uncounted RAY frames walked in
// pixel tiles: RC_TRACE_PACKETS = 2 (default) for camera frames and caller
// ray frames, 1 for camera frames only, 0 never (read once). On the 1080p
// heightfield the primary rays of an 8x4-pixel tile take 0.302 ms this way
// against 0.327 ms per lane, and the caller-ray frame through host memory
// gains 3 %. A caller frame whose neighbouring rays are not coherent would
// lose instead (mode 1). Shadow rays stay per lane: each stops at its first
// occluder, and the warp-wide walk of the union of their paths measured 1.8x
// slower (0.306 vs 0.172 ms).
int trace_packets()
{
    static const int mode = [] {
        const char* v = std::getenv("RC_TRACE_PACKETS");
        return v && v[0] >= '0' && v[0] <= '2' ? int(v[0] - '0') : 2;
    }();
    return mode;
}

// Whether a pixel range is whole lines from the film's first on.
bool whole_lines(uint64_t pixelStart, int64_t count, int64_t width)
{
    return pixelStart == 0 && (count / width) * width == count;
}

// The tiles of a frame (device_types.h), or none: camera rays of any pixel
// range, or one caller ray per pixel of a whole image (other ray lists are
// walked in order: nothing says that a ray's neighbour in the next line is
// near it).
FilmTiles frame_tiles(const rc_ray* rays, uint64_t pixelStart, int64_t count, int64_t width)
{
    if (!RC_TRACE_TILES || width <= 0 || (rays && !whole_lines(pixelStart, count, width)))
        return FilmTiles{};
    return film_tiles(pixelStart, count, width);
}

// Whether an uncounted frame of tiles is walked by packets: whole lines, and
// any range in reference order, where a packet meets each ray's triangles in
// the ray's order. Nearest-first, a packet's order can decide between hits
// that rounding puts before their boxes (33 of 480,000 pixels in a room of
// overlapping coplanar triangles): a range keeps its rays' own walks, and so
// its records do not depend on where it ends.
bool packet_frame(uint64_t pixelStart, int64_t count, int64_t width, int order)
{
    return order == ORDER_REF || whole_lines(pixelStart, count, width);
}

// The tiles of a frame that groups of lanes do not walk. Ranges walked one ray
// per lane take them from four tiles per resident warp on: with fewer the
// longest tile's chain of walks is longer than the longest row's. In order ->
// tiles, device time of ranges of 192k, 240k, 320k, 433k, 607k, 780k and 1.87M
// pixels, 1M triangles: 115 / 125 / 125 / 145 / 191 / 265 / 470 -> 134 / 148 /
// 133 / 157 / 192 / 228 / 387 us. Packets in reference order, from one tile per
// warp on: 78k / 90k / 138k pixels 302 / 313 / 323 -> 401 / 381 / 366 us, the
// others 222 / 268 / 226 / 294 / 535 / 737 / 1,310 -> 224 / 281 / 184 / 238 / 387
// / 600 / 803. Two-level
// scenes gain at all sizes but one: 1M + 200 blobs of 20,480 triangles, 60k, 192k,
// 240k, 320k, 433k, 607k and 1.87M pixels 613 / 416 / 541 / 423 / 648 / 866 /
// 2,092 -> 525 / 403 / 602 / 359 / 570 / 780 / 1,646.
FilmTiles walk_tiles(const LaunchInfo& li, const rc_ray* rays, uint64_t pixelStart, int64_t count, int64_t width,
                     int order, bool instanced)
{
    const int64_t warps = int64_t(li.numSMs) * 32;
    if (!instanced && width > 0 && !whole_lines(pixelStart, count, width) &&
        count < warps * 32 * (order == ORDER_REF ? 1 : 4))
        return FilmTiles{};
    return frame_tiles(rays, pixelStart, count, width);
}

// Sign octant of the shadow rays' direction L for slab_oct (bit k: component
// k negative), or -1 where a component is zero, not finite or too small for
// its reciprocal to be finite (the general box test then applies).
int light_octant(float3 L)
{
    const float c[3] = { L.x, L.y, L.z };
    int oct = 0;
    for (int k = 0; k < 3; ++k)
    {
        if (!std::isfinite(c[k]) || !(std::fabs(c[k]) > 1e-30f))
            return -1;
        if (c[k] < 0.0f)
            oct |= 1 << k;
    }
    return oct;
}

#define RC_FUSED_ARGS li, sc, cam, rays, pixelStart, count, width, tiles, castShadow, L, off, out, queue, ctl

// The one-kernel RAY frame, its shadow walk specialised to the light's
// octant SOCT (or general, -1).
template <int ORDER, bool PACKET, bool INST, bool SL, int SOCT>
cudaError_t launch_fused(const LaunchInfo& li, const DevScene& sc, const DevCamera& cam, const rc_ray* rays,
                         uint64_t pixelStart, int64_t count, int64_t width, FilmTiles tiles,
                         int castShadow, float3 L, float off, rc_cast_pixel* out, int* queue, DevControl* ctl)
{
    auto kf = k_raycast_primary<ORDER, false, PACKET, INST, true, SL, SOCT>;
    static OccupancyCache occF;
    kf<<<persistent_blocks(kf, li.numSMs, occF), kBlock, 0, li.stream>>>(sc, cam, rays, pixelStart, count, width,
                                                                         tiles, castShadow, out, queue, ctl,
                                                                         L, off, nullptr);
    return cudaGetLastError();
}

template <int ORDER, bool COUNT, bool PACKET, bool INST, bool SL = false, bool FUSED = false>
cudaError_t raycast_t(const LaunchInfo& li, const DevScene& sc, const DevCamera& cam, const rc_ray* rays,
                      uint64_t pixelStart, int64_t count, int64_t width, int castShadow, float3 L, float off,
                      rc_cast_pixel* out, int* queue, DevControl* ctl, cudaEvent_t between, float4* origins,
                      int& kernels)
{
    // only the order the warps take the pixels in
    const FilmTiles tiles = walk_tiles(li, rays, pixelStart, count, width, ORDER, INST);
    if (FUSED && castShadow)
    {
        kernels = 1;
        if constexpr (!INST && !SL)
        {
            switch (light_octant(L))
            {
            case 0: return launch_fused<ORDER, PACKET, INST, SL, 0>(RC_FUSED_ARGS);
            case 1: return launch_fused<ORDER, PACKET, INST, SL, 1>(RC_FUSED_ARGS);
            case 2: return launch_fused<ORDER, PACKET, INST, SL, 2>(RC_FUSED_ARGS);
            case 3: return launch_fused<ORDER, PACKET, INST, SL, 3>(RC_FUSED_ARGS);
            case 4: return launch_fused<ORDER, PACKET, INST, SL, 4>(RC_FUSED_ARGS);
            case 5: return launch_fused<ORDER, PACKET, INST, SL, 5>(RC_FUSED_ARGS);
            case 6: return launch_fused<ORDER, PACKET, INST, SL, 6>(RC_FUSED_ARGS);
            case 7: return launch_fused<ORDER, PACKET, INST, SL, 7>(RC_FUSED_ARGS);
            default: break;
            }
        }
        return launch_fused<ORDER, PACKET, INST, SL, -1>(RC_FUSED_ARGS);
    }
    auto kp = k_raycast_primary<ORDER, COUNT, PACKET, INST>;
    auto ks = k_raycast_shadow<COUNT, INST, SL>;
    static OccupancyCache occP, occS;
    kp<<<persistent_blocks(kp, li.numSMs, occP), kBlock, 0, li.stream>>>(sc, cam, rays, pixelStart, count, width, tiles, castShadow, out, queue,
                                     ctl, L, off, castShadow ? origins : nullptr);
    kernels = 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !castShadow)
        return e;
    if (between)
        e = cudaEventRecord(between, li.stream);
    if (e != cudaSuccess)
        return e;
    ks<<<persistent_blocks(ks, li.numSMs, occS), kBlock, 0, li.stream>>>(sc, cam, rays, pixelStart, width, L, off, out, queue, ctl, origins);
    kernels = 2;
    return cudaGetLastError();
}

// Whether uncounted RAY frames trace each shadow ray in the primary kernel
// (k_raycast_primary FUSED); RC_TRACE_FUSED=0 keeps the two kernels with the
// compacted shadow queue (read once).
bool fused_frames()
{
    static const bool on = [] {
        const char* v = std::getenv("RC_TRACE_FUSED");
        return !(v && v[0] == '0');
    }();
    return on;
}

template <int ORDER>
cudaError_t raycast_group(const LaunchInfo& li, const DevScene& sc, const DevCamera& cam, const rc_ray* rays,
                          uint64_t pixelStart, int64_t count, int64_t width, int castShadow, float3 L, float off,
                          rc_cast_pixel* out, DevControl* ctl, bool& taken)
{
    auto k = k_raycast_group<ORDER>;
    static OccupancyCache occ;
    const int blocks = persistent_blocks(k, li.numSMs, occ);
    const unsigned G = frame_group_lanes(sc, count, blocks);
    taken = G != 0u;
    if (!taken)
        return cudaSuccess;
    const FilmTiles tiles = frame_tiles(rays, pixelStart, count, width);
    k<<<blocks, kBlock, 0, li.stream>>>(sc, cam, rays, pixelStart, count, width, tiles, castShadow, out, ctl, L,
                                        off, G, sc.depth);
    return cudaGetLastError();
}

// Uncounted frames: the fused or the two-kernel form.
template <int ORDER, bool PACKET, bool INST, bool SL = false>
cudaError_t raycast_u(const LaunchInfo& li, const DevScene& sc, const DevCamera& cam, const rc_ray* rays,
                      uint64_t pixelStart, int64_t count, int64_t width, int castShadow, float3 L, float off,
                      rc_cast_pixel* out, int* queue, DevControl* ctl, cudaEvent_t between, float4* origins,
                      int& kernels)
{
    return fused_frames() ? raycast_t<ORDER, false, PACKET, INST, SL, true>(li, sc, cam, rays, pixelStart, count,
                                                                             width, castShadow, L, off, out, queue,
                                                                             ctl, between, origins, kernels)
                          : raycast_t<ORDER, false, PACKET, INST, SL, false>(li, sc, cam, rays, pixelStart, count,
                                                                              width, castShadow, L, off, out, queue,
                                                                              ctl, between, origins, kernels);
}

}  // namespace

// Whether the reference-order queries of uncounted frames (the RAY frame's
// shadow rays, rc_cast in RC_ORDER_REFERENCE) take the stackless walk over
// the rope records (RC_STACKLESS=1; read once). The same hits.
bool stackless_walk()
{
    static const bool on = [] {
        const char* v = std::getenv("RC_STACKLESS");
        return v && v[0] == '1';
    }();
    return on;
}

namespace
{

// Rays above which a cast looks at its rays first (cast_large), and nearest-first
// casts walk the 4-wide tree: four per lane of 32 resident warps per SM, eight
// for scenes below 2^15 triangles and in reference order. Below, the gain of
// phases is within what looking costs (10 us for two more launches), or what a
// frame's rays would lose: 400k of them from above, 8,930 triangles: 57 -> 66 us
// nearest-first, 59 -> 66 any hit (from 2^15 triangles on 89 -> 89).
int64_t large_line(const LaunchInfo& li, const DevScene& sc, bool reference)
{
    return int64_t(li.numSMs) * 32 * 32 * (reference || scene_bits(sc) < 15 ? 8 : 4);
}

}  // namespace

int64_t cast_wide_rays(const LaunchInfo& li, const DevScene& sc, int64_t n, int anyHit, int order)
{
    if (anyHit || order != ORDER_NEAREST || li.counting || sc.numInstances > 0 || (sc.ropes && stackless_walk()))
        return 0;
    return std::max<int64_t>(0, n - large_line(li, sc, false));
}

cudaError_t launch_cast(const LaunchInfo& li, const DevScene& sc, const rc_ray* rays, int64_t n, int anyHit,
                        int order, rc_hit* hits, DevControl* ctl)
{
    if (n <= 0)
        return cudaSuccess;
    const bool sl = !li.counting && sc.numInstances == 0 && sc.ropes && stackless_walk();
    if (!li.counting && sc.numInstances == 0 && !sl)
    {
        bool taken = false;
        const cudaError_t e =
            anyHit                   ? cast_group<true, ORDER_REF>(li, sc, rays, n, hits, ctl, taken)
            : order == ORDER_NEAREST ? cast_group<false, ORDER_NEAREST>(li, sc, rays, n, hits, ctl, taken)
                                     : cast_group<false, ORDER_REF>(li, sc, rays, n, hits, ctl, taken);
        if (taken)
            return e;
        const bool large = n > large_line(li, sc, !anyHit && order == ORDER_REF);
        if (anyHit && (large || scene_bits(sc) >= 15))
            return large ? cast_large<true, ORDER_REF>(li, sc, rays, n, hits, ctl)
                         : cast_phased<true, ORDER_REF>(li, sc, rays, n, hits, ctl);
        if (!anyHit && order == ORDER_REF)
            return large ? cast_large<false, ORDER_REF>(li, sc, rays, n, hits, ctl)
                         : cast_phased<false, ORDER_REF>(li, sc, rays, n, hits, ctl);
        if (!anyHit && sc.wide && large)
            return cast_large<false, ORDER_NEAREST>(li, sc, rays, n, hits, ctl);
    }
    if (anyHit)
        return li.counting ? cast_t<true, ORDER_REF, true>(li, sc, rays, n, hits, ctl)
               : sl        ? cast_t<true, ORDER_REF, false, true>(li, sc, rays, n, hits, ctl)
                           : cast_t<true, ORDER_REF, false>(li, sc, rays, n, hits, ctl);
    if (order == ORDER_NEAREST)
        return li.counting ? cast_t<false, ORDER_NEAREST, true>(li, sc, rays, n, hits, ctl)
                           : cast_t<false, ORDER_NEAREST, false>(li, sc, rays, n, hits, ctl);
    return li.counting ? cast_t<false, ORDER_REF, true>(li, sc, rays, n, hits, ctl)
           : sl        ? cast_t<false, ORDER_REF, false, true>(li, sc, rays, n, hits, ctl)
                       : cast_t<false, ORDER_REF, false>(li, sc, rays, n, hits, ctl);
}

cudaError_t launch_raycast(const LaunchInfo& li, const DevScene& sc, const DevCamera& cam, const rc_ray* rays,
                           uint64_t pixelStart, int64_t count, int64_t width, int order, int castShadow,
                           float3 dirToLight, float rayStartOffset, rc_cast_pixel* out, int* shadowQueue,
                           DevControl* ctl, cudaEvent_t between, float4* shadowOrigins, int* kernels)
{
    int launched = 0;
    if (!kernels)
        kernels = &launched;
    *kernels = 0;
    if (count <= 0)
        return cudaSuccess;
#define RC_RAYCAST_ARGS li, sc, cam, rays, pixelStart, count, width, castShadow, dirToLight, rayStartOffset, out, \
                        shadowQueue, ctl, between, shadowOrigins, *kernels
    // two-level scenes: the top level nearest-first, like rc_cast's
    if (sc.numInstances > 0)
        return li.counting ? raycast_t<ORDER_NEAREST, true, false, true>(RC_RAYCAST_ARGS)
                           : raycast_u<ORDER_NEAREST, false, true>(RC_RAYCAST_ARGS);
    if (li.counting)
        return order == ORDER_NEAREST ? raycast_t<ORDER_NEAREST, true, false, false>(RC_RAYCAST_ARGS)
                                      : raycast_t<ORDER_REF, true, false, false>(RC_RAYCAST_ARGS);
    if (fused_frames() && !(stackless_walk() && sc.ropes))
    {
        bool taken = false;
        const cudaError_t e =
            order == ORDER_NEAREST
                ? raycast_group<ORDER_NEAREST>(li, sc, cam, rays, pixelStart, count, width, castShadow, dirToLight,
                                               rayStartOffset, out, ctl, taken)
                : raycast_group<ORDER_REF>(li, sc, cam, rays, pixelStart, count, width, castShadow, dirToLight,
                                           rayStartOffset, out, ctl, taken);
        if (taken)
        {
            *kernels = 1;
            return e;
        }
    }
    const int packets = trace_packets();
    const bool packet = walk_tiles(li, rays, pixelStart, count, width, order, false).columns > 0 &&
                        packet_frame(pixelStart, count, width, order) && (packets == 2 || (packets == 1 && !rays));
    if (stackless_walk() && sc.ropes)
    {
        if (packet)
            return order == ORDER_NEAREST ? raycast_u<ORDER_NEAREST, true, false, true>(RC_RAYCAST_ARGS)
                                          : raycast_u<ORDER_REF, true, false, true>(RC_RAYCAST_ARGS);
        return order == ORDER_NEAREST ? raycast_u<ORDER_NEAREST, false, false, true>(RC_RAYCAST_ARGS)
                                      : raycast_u<ORDER_REF, false, false, true>(RC_RAYCAST_ARGS);
    }
    if (packet)
        return order == ORDER_NEAREST ? raycast_u<ORDER_NEAREST, true, false>(RC_RAYCAST_ARGS)
                                      : raycast_u<ORDER_REF, true, false>(RC_RAYCAST_ARGS);
    return order == ORDER_NEAREST ? raycast_u<ORDER_NEAREST, false, false>(RC_RAYCAST_ARGS)
                                  : raycast_u<ORDER_REF, false, false>(RC_RAYCAST_ARGS);
#undef RC_RAYCAST_ARGS
}

}  // namespace rcx
