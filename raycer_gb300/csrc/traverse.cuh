// BVH traversal of the flat SAH BVH (device side).
//
// The reference traverses with an explicit stack: pop a node; a leaf tests
// its triangles in order; an inner node tests the right child's box and
// pushes it, then the left child's box and pushes it, so the left subtree is
// finished first (FlatBVH::intersect FlatBVH.cpp:22-75, intersectBVH
// intersections.cl:98-148). The root's own box is never tested.
//
// Here the node is the 64-B two-child record of device_types.h, so one fetch
// tests both children:
//   ORDER_REF      descend left, push right (the reference's visit order;
//                  the same boxes are tested, the same triangles in the same
//                  order, the same closest hit — ties to the later triangle,
//                  Triangle.cpp:93 `t > distance` rejects only farther hits).
//   ORDER_NEAREST  descend into the nearer child, push the farther one with
//                  its entry distance, and skip boxes whose entry distance is
//                  beyond the current closest hit. The accepted hit is the
//                  same: minimum t, ties resolved to the larger BVH-order
//                  slot, which is what the reference's order yields.
// Any-hit (shadow rays: isShadowRay + fastOcclusion) always uses the
// reference order and stops at the first triangle found; triangles whose
// material is nonShadowing are skipped (Triangle.cpp:55).
//
// `skip` names the triangle a secondary ray leaves from (-1 for none). Its
// origin is the hit point moved by rayStartOffset along the ray direction, so
// in exact arithmetic the ray travels away from that triangle's plane and
// cannot hit it; in float32 the hit point's rounding (about 1e-6 at
// coordinates of 10) can exceed the 1e-5 offset at grazing angles and report
// the ray's own triangle. Skipping it gives the float64 reference's answer.
#pragma once

#include <cfloat>

#include "rc_math.cuh"

namespace rcx
{

enum TraversalOrder
{
    ORDER_REF = 0,
    ORDER_NEAREST = 1,
    ORDER_WIDE = 2  // kernels only: ORDER_NEAREST's closest hit through the 4-wide BVH (traverse_wide)
};

struct HitF
{
    int slot;  // BVH-order triangle slot, -1 = none
    float t;
    float u;
    float v;
    int inst;  // instance of the hit in a two-level scene, else -1
};

struct TravCount
{
    uint32_t nodes;  // inner nodes fetched (child-pair box tests)
    uint32_t tris;   // triangle tests
};

// 32 bytes of read-only memory (32-byte aligned) as one load: an L1 request
// per lane instead of two.
__device__ __forceinline__ void ldg32(const void* p, float4& a, float4& b)
{
    unsigned long long x, y, z, w;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(x), "=l"(y), "=l"(z), "=l"(w) : "l"(p));
    a = make_float4(__uint_as_float(uint32_t(x)), __uint_as_float(uint32_t(x >> 32)), __uint_as_float(uint32_t(y)),
                    __uint_as_float(uint32_t(y >> 32)));
    b = make_float4(__uint_as_float(uint32_t(z)), __uint_as_float(uint32_t(z >> 32)), __uint_as_float(uint32_t(w)),
                    __uint_as_float(uint32_t(w >> 32)));
}

// Items of `count` pixels in tiles (the tiles' pixels outside the range too).
__device__ __forceinline__ int64_t tile_items(const FilmTiles& t, int64_t count)
{
    return t.columns > 0 ? int64_t(t.columns) * t.rows * 32 : count;
}

// Whether an item is a pixel of the range, and which (in `i`, from the range's
// first). Tiles lie on the film's columns, so that a warp's pixels are one
// tile whatever the width: in a permutation without padding, whose warps
// straddle two tiles where the width is no multiple of 8, the RAY frame of
// 1919x1079 pixels took 544 us instead of 502.
__device__ __forceinline__ bool tile_pixel(const FilmTiles& t, int64_t count, int64_t item, int64_t& i)
{
    i = item;
    if (t.columns > 0)
    {
        const int tile = int(item >> 5);
        const int row = tile / t.columns;
        const int x = (tile - row * t.columns) * 8 + int(item & 7);
        const int64_t y = int64_t(row) * 4 + int((item >> 3) & 3);
        i = y * t.width + x - t.skip;
        if (x >= t.width)
            return false;
    }
    return i >= 0 && i < count;
}

__device__ __forceinline__ void load_node(const DevNode* __restrict__ nodes, int i, float4& a, float4& b, float4& c,
                                          int4& l)
{
    const float4* p = reinterpret_cast<const float4*>(nodes + i);
    a = __ldg(p + 0);
    b = __ldg(p + 1);
    c = __ldg(p + 2);
    l = __ldg(reinterpret_cast<const int4*>(p + 3));
}

// The test of one leaf triangle in traverse(): nonShadowing triangles are
// skipped by any-hit rays (Triangle.cpp:55); returns true when an any-hit
// ray has found its occluder (the walk ends), else updates the closest hit
// (the reference order keeps the later of equal distances, nearest-first
// the larger slot).
template <bool ANY_HIT, int ORDER, bool COUNT>
__device__ __forceinline__ bool leaf_test(const RayF& ray, HitF& hit, bool& found, TravCount& cnt, int slot, int skip,
                                          const float4& ta, const float4& tb, const float4& tc)
{
    if (slot == skip)
        return false;
    if (ANY_HIT && (__float_as_uint(tc.y) & kMetaNonShadowing))
        return false;
    if (COUNT)
        cnt.tris++;
    float t, u, v;
    if (!tri_hit(ray, v3(ta.x, ta.y, ta.z), v3(ta.w, tb.x, tb.y), v3(tb.z, tb.w, tc.x), t, u, v))
        return false;
    if (ANY_HIT)
    {
        hit.slot = slot;
        hit.t = t;
        hit.u = u;
        hit.v = v;
        return true;
    }
    const bool take = ORDER == ORDER_REF ? !(t > hit.t) : (t < hit.t || (t == hit.t && slot > hit.slot));
    if (take)
    {
        hit.slot = slot;
        hit.t = t;
        hit.u = u;
        hit.v = v;
        found = true;
    }
    return false;
}

// Returns true if any triangle was accepted. `hit` must be initialised by
// the caller (slot -1, t = FLT_MAX for a fresh query). `err` is set to 1 on
// a stack overflow (the ray is then abandoned; the host reports it).
// OCT >= 0: the caller guarantees that the ray's inverse direction is finite
// with those signs (ray_octant), and the box tests take slab_oct<OCT>.
template <bool ANY_HIT, int ORDER, bool COUNT, int OCT = -1>
__device__ __forceinline__ bool traverse(const DevScene& sc, const RayF& ray, HitF& hit, TravCount& cnt, int& err,
                                         int skip = -1)
{
    int stack[kMaxStack];
    float sdist[ORDER == ORDER_NEAREST && !ANY_HIT ? kMaxStack : 1];
    int sp = 0;
    int cur = sc.rootLink;
    bool found = false;

    while (true)
    {
        if (cur >= 0)
        {
            float4 a, b, c;
            int4 l;
            load_node(sc.nodes, cur, a, b, c, l);
            if (COUNT)
                cnt.nodes++;
            float e0, e1;
            bool h0, h1;
            if (OCT >= 0)
            {
                h0 = slab_oct<OCT < 0 ? 0 : OCT>(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab_oct<OCT < 0 ? 0 : OCT>(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
#ifndef RC_EXACT_SLAB_ONLY
            else if (ray.finite)
#else
            else if (false)
#endif
            {
                h0 = slab_finite(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab_finite(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
            else
            {
                h0 = slab(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
            if (ORDER == ORDER_NEAREST && !ANY_HIT)
            {
                h0 = h0 && !(e0 > hit.t);
                h1 = h1 && !(e1 > hit.t);
            }
            if (h0 && h1)
            {
                int nearC = l.x, farC = l.y;
                float farD = e1;
                if (ORDER == ORDER_NEAREST && !ANY_HIT && e1 < e0)
                {
                    nearC = l.y;
                    farC = l.x;
                    farD = e0;
                }
                if (sp >= kMaxStack)
                {
                    err = 1;
                    return found;
                }
                stack[sp] = farC;
                if (ORDER == ORDER_NEAREST && !ANY_HIT)
                    sdist[sp] = farD;
                sp++;
                cur = nearC;
                continue;
            }
            if (h0)
            {
                cur = l.x;
                continue;
            }
            if (h1)
            {
                cur = l.y;
                continue;
            }
        }
        else
        {
            int leaf = ~cur;
            int start = leaf >> kLeafCountBits;
            int count = leaf & ((1 << kLeafCountBits) - 1);
            if (!ANY_HIT && ORDER == ORDER_NEAREST)
            {
                // closest hit, nearest-first: two triangles fetched per step
                // (the accepted hit does not depend on the test order; 8 %
                // less time for rc_cast's random rays). Any-hit and
                // reference-order walks keep one triangle per step: in the
                // issue-bound RAY frame the pairs cost more than they hid.
                for (int i = 0; i < count; i += 2)
                {
                    const int s0 = start + i;
                    const int s1 = start + min(i + 1, count - 1);
                    const float4* p0 = reinterpret_cast<const float4*>(sc.tris + s0);
                    const float4* p1 = reinterpret_cast<const float4*>(sc.tris + s1);
                    const float4 a0 = __ldg(p0 + 0), b0 = __ldg(p0 + 1), c0 = __ldg(p0 + 2);
                    const float4 a1 = __ldg(p1 + 0), b1 = __ldg(p1 + 1), c1 = __ldg(p1 + 2);
                    leaf_test<ANY_HIT, ORDER, COUNT>(ray, hit, found, cnt, s0, skip, a0, b0, c0);
                    if (i + 1 < count)
                        leaf_test<ANY_HIT, ORDER, COUNT>(ray, hit, found, cnt, s1, skip, a1, b1, c1);
                }
            }
            else
            {
                for (int i = 0; i < count; ++i)
                {
                    const int slot = start + i;
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + slot);
                    if (slot != skip && leaf_test<ANY_HIT, ORDER, COUNT>(ray, hit, found, cnt, slot, skip,
                                                                         __ldg(tp + 0), __ldg(tp + 1), __ldg(tp + 2)))
                        return true;
                }
            }
        }

        // pop
        while (true)
        {
            if (sp == 0)
                return found;
            sp--;
            cur = stack[sp];
            if (ORDER == ORDER_NEAREST && !ANY_HIT && sdist[sp] > hit.t)
                continue;
            break;
        }
    }
}

// The reference's order without a stack, on the rope records (DevRope,
// every child box of the binary tree once, in the reference's preorder): a
// hit inner box continues at the next record (its left child), a hit leaf
// box's triangles are tested in order, and after a leaf or on a miss the
// walk jumps to the record after the box's subtree. Each ray meets the boxes
// and triangles of traverse<ANY_HIT, ORDER_REF> in the same order (the same
// slab test on the same float boxes), so it returns the same closest hit
// (ties to the later triangle) or the same first any-hit; one 32-byte record
// per tested box, no stack, and a descent reads the next record in memory.
// Needs sc.ropes (callers fall back to traverse() without them).
template <bool ANY_HIT>
__device__ __forceinline__ bool test_leaf(const DevScene& sc, const RayF& ray, HitF& hit, int leafCode, int skip,
                                          bool& found)
{
    const int leaf = ~leafCode;
    const int start = leaf >> kLeafCountBits;
    const int count = leaf & ((1 << kLeafCountBits) - 1);
    for (int i = 0; i < count; ++i)
    {
        const int slot = start + i;
        if (slot == skip)
            continue;
        const float4* tp = reinterpret_cast<const float4*>(sc.tris + slot);
        const float4 ta = __ldg(tp + 0);
        const float4 tb = __ldg(tp + 1);
        const float4 tc = __ldg(tp + 2);
        if (ANY_HIT && (__float_as_uint(tc.y) & kMetaNonShadowing))
            continue;
        float t, u, v;
        if (tri_hit(ray, v3(ta.x, ta.y, ta.z), v3(ta.w, tb.x, tb.y), v3(tb.z, tb.w, tc.x), t, u, v) &&
            (ANY_HIT || !(t > hit.t)))
        {
            hit.slot = slot;
            hit.t = t;
            hit.u = u;
            hit.v = v;
            found = true;
            if (ANY_HIT)
                return true;
        }
    }
    return false;
}

template <bool ANY_HIT>
__device__ __forceinline__ bool traverse_stackless(const DevScene& sc, const RayF& ray, HitF& hit, int skip)
{
    bool found = false;
    if (sc.rootLink < 0)
    {
        test_leaf<ANY_HIT>(sc, ray, hit, sc.rootLink, skip, found);  // a leaf root: its triangles only
        return found;
    }
    const int end = sc.ropeCount;
    int r = 0;
    while (r < end)
    {
        const float4* p = reinterpret_cast<const float4*>(sc.ropes + r);
        const float4 a = __ldg(p);
        const float4 b = __ldg(p + 1);  // hi.y, hi.z, link, miss
        float e;
        const bool h = ray.finite ? slab_finite(ray, a.x, a.w, a.y, b.x, a.z, b.y, e)
                                  : slab(ray, a.x, a.w, a.y, b.x, a.z, b.y, e);
        const int link = __float_as_int(b.z);
        if (h && link >= 0)
        {
            ++r;
            continue;
        }
        if (h && test_leaf<ANY_HIT>(sc, ray, hit, link, skip, found))
            return true;
        r = __float_as_int(b.w);
    }
    return found;
}

// Entry distance of one child box of a wide node, or +inf when the ray misses
// it or enters it beyond `limit` (the current closest hit); any ray. NaN where
// slab() hits the box with a NaN entry (see wide_node_step).
__device__ __forceinline__ float wide_entry(const RayF& ray, float lox, float hix, float loy, float hiy, float loz,
                                            float hiz, float limit)
{
    float e;
    const bool h = slab(ray, lox, hix, loy, hiy, loz, hiz, e);
    return h && !(e > limit) ? e : __int_as_float(0x7f800000);
}

// The plane distances of two children on one axis, (plane - o) * inv in
// slab_finite's arithmetic (subtract, then multiply, each rounded), for both
// children at once.
struct AxisF2
{
    F2 no;   // -o, -o
    F2 inv;  // inv, inv
};

__device__ __forceinline__ F2 plane2(float a, float b, const AxisF2& x) { return mul2(add2(f2(a, b), x.no), x.inv); }

// Entry from the plane distances, as wide_entry for a ray whose inverse
// direction is finite: entered at the largest near distance (at least 0),
// left at the smallest far one, both within `limit`.
__device__ __forceinline__ float wide_entry_of(float x0, float x1, float y0, float y1, float z0, float z1, float limit)
{
    const float e = fmaxf(fmax3(fminf(x0, x1), fminf(y0, y1), fminf(z0, z1)), 0.0f);
    const float f = fminf(fmin3(fmaxf(x0, x1), fmaxf(y0, y1), fmaxf(z0, z1)), limit);
    return e <= f ? e : __int_as_float(0x7f800000);
}

// Orders two (distance, link) pairs by distance.
__device__ __forceinline__ void wide_cswap(float& da, int& la, float& db, int& lb)
{
    const bool s = db < da;
    const float d = s ? db : da;
    const int l = s ? lb : la;
    db = s ? da : db;
    lb = s ? la : lb;
    da = d;
    la = l;
}

// Closest hit through the 4-wide BVH (sc.wide; wide_build.cu): one 128-B
// node fetch tests up to four child boxes, the children hit within the
// current closest distance are sorted by entry distance (a five-exchange
// network), the nearest is entered and the others pushed farthest first with
// their entry distances, and pops skip entries beyond the current hit. The
// leaves and their triangle tests are the binary tree's, and the accepted
// hit (minimum t, ties to the larger slot) does not depend on the order, so
// it is traverse<false, ORDER_NEAREST>'s, but for overlapping coplanar
// triangles where rounding puts hits before their boxes (see traverse_group):
// casts walk such rays again, two-level bounces put them aside, and the paths
// of one-level scenes keep this walk's hit (at 500x400, 475-7,495 pixels of
// scenes made of such sheets differ from the counted render's film, none of
// others). Rays whose inverse direction is not
// finite can reach other boxes here than there (see wide_node_step) and walk
// the binary tree. No node or triangle counts: counted frames use the binary
// traversal.
// Where a 4-wide walk stands between steps: the node or leaf link to visit
// next and the stack depth (the stack arrays are the caller's).
struct WideWalk
{
    static constexpr bool kFinite = true;  // only rays whose inverse direction is finite
    int cur;
    int sp;
    __device__ __forceinline__ void abandon();
    // boxes entered beyond this are skipped
    __device__ __forceinline__ float limit(const HitF& hit) const { return hit.t; }
    // the box of `cur` was entered at e; the hit lies in it
    __device__ __forceinline__ void entered(float) {}
    __device__ __forceinline__ void accepted() {}
};

// A walk that is over (no leaf code has this value: a leaf's last triangle
// lies below 2^27).
constexpr int kWalkDone = -0x7fffffff - 1;
// A lane without a walk (no leaf code either: its 14 triangles would start
// at slot 2^27 - 1, the last one).
constexpr int kWalkNone = -0x7fffffff;

// A walk's stack in local memory.
struct LocalStack
{
    static constexpr int kEntries = kMaxStack;
    int2* e;
    static constexpr int kNear = kMaxStack;
    __device__ __forceinline__ void putNear(int i, int2 v) { e[i] = v; }
    __device__ __forceinline__ void put(int i, int2 v) { e[i] = v; }
    __device__ __forceinline__ int2 get(int i) const { return e[i]; }
};

// A walk's stack with its first D entries in shared memory, entry i of the
// block's threads side by side (a warp's accesses meet no bank twice, whatever
// the depths), the rest in local memory.
template <int D, int THREADS, int ENTRIES = kMaxStack, typename Entry = int2>
struct SharedStack
{
    static constexpr int kEntries = ENTRIES;
    static constexpr int kNear = D;
    __device__ __forceinline__ void putNear(int i, Entry v) { near[i * THREADS] = v; }
    Entry* near;  // this thread's entry 0
    Entry* far;
    __device__ __forceinline__ void put(int i, Entry v)
    {
        if (i < D)
            near[i * THREADS] = v;
        else
            far[i - D] = v;
    }
    __device__ __forceinline__ Entry get(int i) const { return i < D ? near[i * THREADS] : far[i - D]; }
    // an entry apart from the stack, where the near entries have a row more
    __device__ __forceinline__ Entry& extra() const { return near[D * THREADS]; }
};

__device__ __forceinline__ void WideWalk::abandon()
{
    sp = 0;
    cur = kWalkDone;
}

// How far past the current closest hit a walk goes that must meet every box
// which could decide a tie (see traverse_group). A margin that was measured, not
// a bound: over 16M rays at coplanar triangles (axis-aligned and tilted planes,
// scales of 0.1-100 at offsets up to 1,000, origins from 1e-7 of the scale above
// the plane on, grazing to 0.1 %) no hit lies more than 0.015 % before the entry
// of its leaf. Axis-aligned planes subtract exactly; the box of a tilted
// triangle is thick where its rounding is large.
constexpr float kTieCull = 1.01f;

// A walk whose hit is reported (rc_cast): it keeps the entry distance of the
// hit's leaf and skips boxes only past kTieCull times the hit.
struct CastWalk
{
    static constexpr bool kFinite = false;  // any ray
    int cur;
    int sp;
    float entry;     // of cur
    float hitEntry;  // of the hit's leaf
    __device__ __forceinline__ void abandon()
    {
        sp = 0;
        cur = kWalkDone;
    }
    __device__ __forceinline__ float limit(const HitF& hit) const { return hit.t * kTieCull; }
    __device__ __forceinline__ void entered(float e) { entry = e; }
    __device__ __forceinline__ void accepted() { hitEntry = entry; }
};

// Pops the next stack entry still within the current hit, or ends the walk.
template <typename Walk, typename Stack>
__device__ __forceinline__ void wide_pop(const HitF& hit, Walk& w, const Stack& stack)
{
    while (w.sp > 0)
    {
        const int2 e = stack.get(--w.sp);
        w.cur = e.x;
        if (!(__int_as_float(e.y) > w.limit(hit)))
        {
            w.entered(__int_as_float(e.y));
            return;
        }
    }
    w.cur = kWalkDone;
}

// Whether a walk ended undecided: its ray has to walk the binary trees.
__device__ __forceinline__ bool walk_undecided(const HitF& hit) { return !(hit.t == hit.t); }

// Node step of the 4-wide walk (w.cur >= 0): enters the nearest child hit
// within the current closest distance and pushes the others; with none hit,
// pops. On stack overflow err = 1 and the walk is over.
//
// A direction component of zero with the origin on a box's lower plane makes
// slab()'s product a NaN (0 * inf), and with it, in x, the box's entry: slab()
// then hits the box wherever its other planes lie. So a box inside a parent
// that the ray misses can be hit, and which boxes a ray reaches depends on the
// tree that is walked: the walk ends here, undecided, with the hit's t a NaN.
// (Taken as entered at 0,
// such boxes gave 498 other triangles of 32,768 vertical rays at the vertices
// of a 256x128 heightfield; dropped, 24,677 of its 32,387 hits were lost.)
// Without a NaN entry the boxes reached are the binary walk's, up to boxes
// that are flat in a direction the ray has no part of, whose triangles it
// cannot hit. No triangle accepts a ray that has a NaN itself: it leaves the
// node. The path tracer's walks keep to finite inverse directions: its kernels
// ran 6-10 % slower with this branch and what follows from it.
template <typename Walk, typename Stack>
__device__ __forceinline__ void wide_node_step(const DevNode4* __restrict__ wide, const RayF& ray, HitF& hit, Walk& w,
                                               Stack& stack, int& err)
{
    const float kInf = __int_as_float(0x7f800000);
    const float4* p = reinterpret_cast<const float4*>(wide + w.cur);
    float4 lox, hix, loy, hiy, loz, hiz, lf, mf;
    ldg32(p + 0, lox, hix);
    ldg32(p + 2, loy, hiy);
    ldg32(p + 4, loz, hiz);
    ldg32(p + 6, lf, mf);
    const int4 l = make_int4(__float_as_int(lf.x), __float_as_int(lf.y), __float_as_int(lf.z), __float_as_int(lf.w));
    const int nc = __float_as_int(mf.x);
    const float limit = w.limit(hit);
    float d0, d1, d2, d3;
    if (Walk::kFinite || ray.finite)
    {
        const AxisF2 X{ f2(-ray.o.x, -ray.o.x), f2(ray.inv.x, ray.inv.x) };
        const AxisF2 Y{ f2(-ray.o.y, -ray.o.y), f2(ray.inv.y, ray.inv.y) };
        const AxisF2 Z{ f2(-ray.o.z, -ray.o.z), f2(ray.inv.z, ray.inv.z) };
        {
            const F2 x0 = plane2(lox.x, lox.y, X), x1 = plane2(hix.x, hix.y, X);
            const F2 y0 = plane2(loy.x, loy.y, Y), y1 = plane2(hiy.x, hiy.y, Y);
            const F2 z0 = plane2(loz.x, loz.y, Z), z1 = plane2(hiz.x, hiz.y, Z);
            d0 = wide_entry_of(f2_lo(x0), f2_lo(x1), f2_lo(y0), f2_lo(y1), f2_lo(z0), f2_lo(z1), limit);
            d1 = wide_entry_of(f2_hi(x0), f2_hi(x1), f2_hi(y0), f2_hi(y1), f2_hi(z0), f2_hi(z1), limit);
        }
        {
            const F2 x0 = plane2(lox.z, lox.w, X), x1 = plane2(hix.z, hix.w, X);
            const F2 y0 = plane2(loy.z, loy.w, Y), y1 = plane2(hiy.z, hiy.w, Y);
            const F2 z0 = plane2(loz.z, loz.w, Z), z1 = plane2(hiz.z, hiz.w, Z);
            d2 = wide_entry_of(f2_lo(x0), f2_lo(x1), f2_lo(y0), f2_lo(y1), f2_lo(z0), f2_lo(z1), limit);
            d3 = wide_entry_of(f2_hi(x0), f2_hi(x1), f2_hi(y0), f2_hi(y1), f2_hi(z0), f2_hi(z1), limit);
        }
    }
    else
    {
        d0 = wide_entry(ray, lox.x, hix.x, loy.x, hiy.x, loz.x, hiz.x, limit);
        d1 = wide_entry(ray, lox.y, hix.y, loy.y, hiy.y, loz.y, hiz.y, limit);
        d2 = wide_entry(ray, lox.z, hix.z, loy.z, hiy.z, loz.z, hiz.z, limit);
        d3 = wide_entry(ray, lox.w, hix.w, loy.w, hiy.w, loz.w, hiz.w, limit);
        if (d0 != d0 || d1 != d1 || (nc > 2 && d2 != d2) || (nc > 3 && d3 != d3))
        {
            const V3 o = ray.o, d = ray.d;
            if (o.x != o.x || o.y != o.y || o.z != o.z || d.x != d.x || d.y != d.y || d.z != d.z)
            {
                wide_pop(hit, w, stack);
                return;
            }
            hit.t = __int_as_float(0x7fffffff);
            w.abandon();
            return;
        }
    }
    if (nc < 3)
        d2 = kInf;
    if (nc < 4)
        d3 = kInf;
    int l0 = l.x, l1 = l.y, l2 = l.z, l3 = l.w;
    wide_cswap(d0, l0, d1, l1);
    wide_cswap(d2, l2, d3, l3);
    wide_cswap(d0, l0, d2, l2);
    wide_cswap(d1, l1, d3, l3);
    wide_cswap(d1, l1, d2, l2);
    if (d0 < kInf)
    {
        // room for three in the near entries: no test per entry
        if (w.sp <= Stack::kNear - 3)
        {
            if (d3 < kInf)
                stack.putNear(w.sp++, make_int2(l3, __float_as_int(d3)));
            if (d2 < kInf)
                stack.putNear(w.sp++, make_int2(l2, __float_as_int(d2)));
            if (d1 < kInf)
                stack.putNear(w.sp++, make_int2(l1, __float_as_int(d1)));
            w.cur = l0;
            w.entered(d0);
            return;
        }
        if (w.sp > Stack::kEntries - 3 &&
            w.sp + (d1 < kInf ? 1 : 0) + (d2 < kInf ? 1 : 0) + (d3 < kInf ? 1 : 0) > Stack::kEntries)
        {
            err = 1;
            w.abandon();
            return;
        }
        if (d3 < kInf)
            stack.put(w.sp++, make_int2(l3, __float_as_int(d3)));
        if (d2 < kInf)
            stack.put(w.sp++, make_int2(l2, __float_as_int(d2)));
        if (d1 < kInf)
            stack.put(w.sp++, make_int2(l1, __float_as_int(d1)));
        w.cur = l0;
        w.entered(d0);
        return;
    }
    wide_pop(hit, w, stack);
}

// The closest-hit test of one leaf triangle in the 4-wide walk.
template <typename Walk, typename Stack>
__device__ __forceinline__ void wide_leaf_test(const RayF& ray, HitF& hit, Walk& w, const Stack&, int slot, int skip,
                                               const float4& ta, const float4& tb, const float4& tc)
{
    if (slot == skip)
        return;
    float t, u, v;
    if (tri_hit(ray, v3(ta.x, ta.y, ta.z), v3(ta.w, tb.x, tb.y), v3(tb.z, tb.w, tc.x), t, u, v) &&
        (t < hit.t || (t == hit.t && slot > hit.slot)))
    {
        hit.slot = slot;
        hit.t = t;
        hit.u = u;
        hit.v = v;
        w.accepted();
    }
}

// Leaf step (w.cur < 0): two of the leaf's triangles, both fetched before
// either is tested (the second index clamped to the leaf: an odd leaf fetches
// its last triangle twice and tests it once), then the rest of the leaf as
// the next link, or the pop. The accepted hit does not depend on the order
// of the tests. (Both triangles at once in two-wide arithmetic, from records
// of interleaved pairs: no faster, for 8 more registers and 60 MB per 1M
// triangles.)
template <typename Walk, typename Stack>
__device__ __forceinline__ void wide_leaf_step(const DevTri* __restrict__ tris, const RayF& ray, HitF& hit, Walk& w,
                                               const Stack& stack, int skip)
{
    const int leaf = ~w.cur;
    const int s0 = leaf >> kLeafCountBits;
    const int count = leaf & ((1 << kLeafCountBits) - 1);
    const int s1 = s0 + min(1, count - 1);
    const float4* p0 = reinterpret_cast<const float4*>(tris + s0);
    const float4* p1 = reinterpret_cast<const float4*>(tris + s1);
    const float4 a0 = __ldg(p0 + 0), b0 = __ldg(p0 + 1), c0 = __ldg(p0 + 2);
    const float4 a1 = __ldg(p1 + 0), b1 = __ldg(p1 + 1), c1 = __ldg(p1 + 2);
    wide_leaf_test(ray, hit, w, stack, s0, skip, a0, b0, c0);
    if (count > 1)
        wide_leaf_test(ray, hit, w, stack, s1, skip, a1, b1, c1);
    if (count > 2)
        w.cur = ~(((s0 + 2) << kLeafCountBits) | (count - 2));
    else
        wide_pop(hit, w, stack);
}

// A walk of a two-level scene: the top-level tree over the instances (inst =
// -1) or an instance's mesh, whose entries lie above `base` of one stack. At
// the top level a leaf code names instances.
//
// The hit is that of the binary walk (traverse_instanced) unless its order
// decides, and then the walk ends undecided:
//   the same triangle at the same distance in two instances: the one met
//   first is the hit;
//   a hit before the entry of a box around it (see traverse_group), and
//   another one nearer than that entry: met first, it hides the box.
// To meet such hits the walk skips boxes only past kTieCull times the hit.
constexpr int kWalkReturn = -0x7ffffffe;  // the mesh is done (no leaf code: 13 triangles would start at the last slot)

struct TwoLevelWalk
{
    static constexpr bool kFinite = true;
    int cur;
    int sp;
    int base;
    int inst;
    float entry;  // of cur
    __device__ __forceinline__ void abandon()
    {
        sp = base = 0;
        inst = -1;
        cur = kWalkDone;
    }
    __device__ __forceinline__ float limit(const HitF& hit) const { return hit.t * kTieCull; }
    __device__ __forceinline__ void entered(float e) { entry = e; }
};

// The leaf test of a two-level walk. The stack's extra entry holds the entries
// of the boxes around the hit (x) and of the instance (y).
template <typename Stack>
__device__ __forceinline__ void wide_leaf_test(const RayF& ray, HitF& hit, TwoLevelWalk& w, const Stack& stack, int slot,
                                               int skip, const float4& ta, const float4& tb, const float4& tc)
{
    if (slot == skip)
        return;
    float t, u, v;
    if (!tri_hit(ray, v3(ta.x, ta.y, ta.z), v3(ta.w, tb.x, tb.y), v3(tb.z, tb.w, tc.x), t, u, v))
        return;
    bool undecided;
    if (t < hit.t || (t == hit.t && slot > hit.slot))
    {
        const float e = fmaxf(w.entry, __int_as_float(stack.extra().y));
        undecided = hit.t < e;
        stack.extra().x = __float_as_int(e);
        hit.slot = slot;
        hit.t = t;
        hit.u = u;
        hit.v = v;
    }
    else
        undecided = (t == hit.t && slot == hit.slot) || t < __int_as_float(stack.extra().x);
    if (undecided)
        hit.t = __int_as_float(0x7fffffff);
}

template <typename Stack>
__device__ __forceinline__ void wide_pop(const HitF& hit, TwoLevelWalk& w, const Stack& stack)
{
    while (w.sp > w.base)
    {
        const int2 e = stack.get(--w.sp);
        w.cur = e.x;
        if (!(__int_as_float(e.y) > w.limit(hit)))
        {
            w.entered(__int_as_float(e.y));
            return;
        }
    }
    w.cur = w.inst >= 0 ? kWalkReturn : kWalkDone;
}

// One step of the 4-wide walk, a node's or a leaf's. Returns true when the
// walk is over.
template <typename Stack>
__device__ __forceinline__ bool wide_step(const DevNode4* __restrict__ wide, const DevTri* __restrict__ tris,
                                          const RayF& ray, HitF& hit, WideWalk& w, Stack& stack, int skip, int& err)
{
    if (w.cur >= 0)
        wide_node_step(wide, ray, hit, w, stack, err);
    else
        wide_leaf_step(tris, ray, hit, w, stack, skip);
    return w.cur == kWalkDone;
}

// Steps of the binary tree's walk in the reference's order, for warps that
// take one phase at a time: the boxes and triangles of traverse<ANY_HIT,
// ORDER_REF>, in its order. Stack entries are links.
struct RefWalk
{
    int cur;
    int sp;
};

template <typename Stack>
__device__ __forceinline__ void ref_pop(RefWalk& w, const Stack& stack)
{
    w.cur = w.sp > 0 ? stack.get(--w.sp) : kWalkDone;
}

template <typename Stack>
__device__ __forceinline__ void ref_node_step(const DevNode* __restrict__ nodes, const RayF& ray, RefWalk& w, Stack& stack)
{
    float4 a, b, c, lf;
    ldg32(nodes + w.cur, a, b);
    ldg32(reinterpret_cast<const float4*>(nodes + w.cur) + 2, c, lf);
    const int l0 = __float_as_int(lf.x), l1 = __float_as_int(lf.y);
    float e0, e1;
    bool h0, h1;
    if (ray.finite)
    {
        h0 = slab_finite(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
        h1 = slab_finite(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
    }
    else
    {
        h0 = slab(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
        h1 = slab(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
    }
    if (h0 && h1)
        stack.put(w.sp++, l1);  // no deeper than the tree, which fits the stack (checked at upload)
    if (h0 || h1)
        w.cur = h0 ? l0 : l1;
    else
        ref_pop(w, stack);
}

template <bool ANY_HIT, typename Stack>
__device__ __forceinline__ void ref_leaf_step(const DevTri* __restrict__ tris, const RayF& ray, HitF& hit, RefWalk& w,
                                              const Stack& stack, int skip)
{
    const int leaf = ~w.cur;
    const int s0 = leaf >> kLeafCountBits;
    const int count = leaf & ((1 << kLeafCountBits) - 1);
    const int s1 = s0 + min(1, count - 1);
    const float4* p0 = reinterpret_cast<const float4*>(tris + s0);
    const float4* p1 = reinterpret_cast<const float4*>(tris + s1);
    const float4 a0 = __ldg(p0 + 0), b0 = __ldg(p0 + 1), c0 = __ldg(p0 + 2);
    const float4 a1 = __ldg(p1 + 0), b1 = __ldg(p1 + 1), c1 = __ldg(p1 + 2);
    TravCount none{ 0, 0 };
    bool found = false;
    bool over = leaf_test<ANY_HIT, ORDER_REF, false>(ray, hit, found, none, s0, skip, a0, b0, c0);
    if (!over && count > 1)
        over = leaf_test<ANY_HIT, ORDER_REF, false>(ray, hit, found, none, s1, skip, a1, b1, c1);
    if (over)
        w.cur = kWalkDone;
    else if (count > 2)
        w.cur = ~(((s0 + 2) << kLeafCountBits) | (count - 2));
    else
        ref_pop(w, stack);
}

// The walk of a ray whose inverse direction is finite, to its end.
__device__ __forceinline__ bool traverse_wide(const DevScene& sc, const RayF& ray, HitF& hit, int& err, int skip)
{
    int2 entries[kMaxStack];
    LocalStack stack{ entries };
    WideWalk w{ sc.wideRoot, 0 };
    while (!wide_step(sc.wide, sc.tris, ray, hit, w, stack, skip, err))
    {
    }
    return hit.slot >= 0;
}

// One stack entry of the warp-wide traversal: a node link and the lanes
// whose rays take part in its subtree.
struct PacketEntry
{
    int link;
    unsigned lanes;
};

// Warp-wide (masked packet) closest-hit traversal: the 32 lanes of a warp,
// one ray each, walk one shared node sequence, so every node and triangle
// record is one broadcast load and the control flow stays converged. Must be
// called by all 32 lanes together; `active` marks the lanes with a ray;
// `wstack` is this warp's kMaxStack-entry stack in shared memory. Each lane
// makes the tests its own traverse() call would make, in the same order:
//   ORDER_REF      the shared sequence is the tree's preorder restricted to
//                  the boxes some lane hits (left subtree first); a lane takes
//                  part only in the subtrees whose box its ray hits, so it
//                  meets its triangles in its per-ray order and gets the same
//                  closest hit (ties to the later triangle).
//   ORDER_NEAREST  the warp descends first into the child that most of its
//                  lanes find nearer; each lane culls boxes whose entry
//                  distance lies beyond its own current hit. The accepted hit
//                  (minimum t, ties to the larger slot) does not depend on
//                  the order, but where rounding puts hits on overlapping
//                  coplanar triangles before their boxes (see traverse_group).
// It pays for coherent rays (the primary rays of a pixel tile); any-hit
// shadow rays, which stop at different depths, ran slower this way than one
// traversal per lane. Node and triangle counts are not kept: counted frames
// use traverse().
template <int ORDER>
__device__ __forceinline__ bool traverse_packet(const DevScene& sc, const RayF& ray, HitF& hit, int& err, int skip,
                                                bool active, PacketEntry* __restrict__ wstack)
{
    constexpr bool CULL = ORDER == ORDER_NEAREST;
    constexpr unsigned kAll = 0xffffffffu;
    float sdist[CULL ? kMaxStack : 1];  // this lane's entry distance of each stacked box
    const unsigned bit = 1u << (threadIdx.x & 31u);
    bool found = false;
    int sp = 0;
    int cur = sc.rootLink;
    unsigned curMask = __ballot_sync(kAll, active);
    if (curMask == 0)
        return false;

    while (true)
    {
        if (cur >= 0)
        {
            float4 a, b, c;
            int4 l;
            load_node(sc.nodes, cur, a, b, c, l);
            float e0 = 0.0f, e1 = 0.0f;
            bool h0 = false, h1 = false;
            if (curMask & bit)
            {
                if (ray.finite)
                {
                    h0 = slab_finite(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                    h1 = slab_finite(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
                }
                else
                {
                    h0 = slab(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                    h1 = slab(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
                }
                if (CULL)
                {
                    h0 = h0 && !(e0 > hit.t);
                    h1 = h1 && !(e1 > hit.t);
                }
            }
            const unsigned m0 = __ballot_sync(kAll, h0);
            const unsigned m1 = __ballot_sync(kAll, h1);
            if (m0 && m1)
            {
                bool rightFirst = false;
                if (CULL)
                {
                    const unsigned vote = __ballot_sync(kAll, h0 && h1 && e1 < e0);
                    rightFirst = 2 * __popc(vote) > __popc(m0 & m1);
                }
                if (sp >= kMaxStack)
                {
                    err = 1;
                    return found;
                }
                __syncwarp();  // every lane has read the entry this push may replace
                if ((threadIdx.x & 31u) == 0)
                    wstack[sp] = PacketEntry{ rightFirst ? l.x : l.y, rightFirst ? m0 : m1 };
                if (CULL)
                    sdist[sp] = rightFirst ? e0 : e1;
                sp++;
                cur = rightFirst ? l.y : l.x;
                curMask = rightFirst ? m1 : m0;
                continue;
            }
            if (m0 | m1)
            {
                cur = m0 ? l.x : l.y;
                curMask = m0 | m1;
                continue;
            }
        }
        else
        {
            const int leaf = ~cur;
            const int start = leaf >> kLeafCountBits;
            const int count = leaf & ((1 << kLeafCountBits) - 1);
            const bool in = (curMask & bit) != 0;
            TravCount none{ 0, 0 };
            for (int i = 0; i < count; ++i)
            {
                const int slot = start + i;
                const float4* tp = reinterpret_cast<const float4*>(sc.tris + slot);
                const float4 ta = __ldg(tp + 0);
                const float4 tb = __ldg(tp + 1);
                const float4 tc = __ldg(tp + 2);
                if (in)
                    leaf_test<false, ORDER, false>(ray, hit, found, none, slot, skip, ta, tb, tc);
            }
        }

        // pop the next subtree some lane still takes part in
        while (true)
        {
            if (sp == 0)
                return found;
            sp--;
            __syncwarp();
            const PacketEntry e = wstack[sp];
            bool in = (e.lanes & bit) != 0;
            if (CULL && in && sdist[sp] > hit.t)
                in = false;
            curMask = __ballot_sync(kAll, in);
            cur = e.link;
            if (curMask)
                break;
        }
    }
}

// One ray walked by a group of G lanes (a power of two, 4..32): calls with
// fewer rays than the GPU has lanes are bound by the latency of one ray's
// walk, a chain of dependent node fetches (a grazing ray over 1M triangles
// visits hundreds), while most lanes have no ray. The group's lanes pop up to
// G entries of one shared stack at a time, so that many nodes and leaves of
// the ray are in flight together. All 32 lanes of a warp call this together,
// the lanes of a group with the same ray; `active`: the group has a ray.
// `stack`: the group's entries (link, entry distance) in shared memory,
// `capacity` of them. A pop of G entries can push 2 G; once fewer than
// `reserve` (at least the tree's depth) + G would be left, the group goes on
// one entry at a time, depth first, which needs no more than the reserve.
// The result (in every lane of the group) is the one-lane walk's:
//   any-hit       the reference's first occluder is the one in the smallest
//                 slot (the reference order meets leaves in slot order);
//   closest hit   the minimum t, ties to the larger slot, does not depend on
//                 the order the boxes are met in, with two exceptions, which
//                 the group's first lane walks again alone. ORDER_REF takes
//                 every NaN distance it meets (rays or vertices with NaN, or
//                 so large that products overflow). ORDER_NEAREST skips a box
//                 entered beyond the current hit, and rounding can put a
//                 box's entry behind a hit inside it (overlapping coplanar
//                 triangles): if the winner lies before its own leaf's entry,
//                 the order may have decided; if not, no walk can have skipped
//                 it (entries grow downward, hits only come nearer). The
//                 group itself skips boxes only past kTieCull times the
//                 current hit, so that it meets such winners.

template <int ORDER>
static __device__ __noinline__ bool traverse_alone(const DevScene& sc, const RayF& ray, HitF& hit, int skip)
{
    TravCount none{ 0, 0 };
    int err = 0;  // the tree's depth is within the stack (checked at upload)
    hit = HitF{ -1, FLT_MAX, 0.0f, 0.0f, -1 };
    return traverse<false, ORDER, false>(sc, ray, hit, none, err, skip);
}

template <bool ANY_HIT, int ORDER>
__device__ __forceinline__ bool traverse_group(const DevScene& sc, const RayF& ray, HitF& hit, int skip, bool active,
                                               unsigned G, int2* __restrict__ stack, int capacity, int reserve)
{
    constexpr unsigned kAll = 0xffffffffu;
    constexpr bool CULL = !ANY_HIT && ORDER == ORDER_NEAREST;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned gl = lane & (G - 1u);           // lane within the group
    const unsigned shift = lane & ~(G - 1u);       // first lane of the group
    const unsigned gmask = kAll >> (32u - G);      // the group's lanes, shifted down
    const unsigned below = (1u << gl) - 1u;
    const int limit = capacity - reserve - int(G); // most entries before a pop of G
    float cull = __int_as_float(0x7f800000);       // boxes entered beyond this are skipped
    int count = 0;
    float he = 0.0f;                               // entry distance of the hit's leaf
    bool odd = false;                              // reference order: a NaN distance was met
    bool found = false;
    if (active)
    {
        count = 1;
        if (gl == 0)
            stack[0] = make_int2(sc.rootLink, 0);
    }
    __syncwarp();
    while (__ballot_sync(kAll, count > 0))
    {
        const int pops = count > limit ? min(count, 1) : min(count, int(G));
        bool mine = int(gl) < pops;
        int2 e = make_int2(0, 0);
        if (mine)
            e = stack[count - 1 - int(gl)];
        count -= pops;
        __syncwarp();  // every lane has read its entry before the pushes below
        if (CULL && __int_as_float(e.y) > cull)
            mine = false;
        bool hNear = false, hFar = false;
        int nearC = 0, farC = 0;
        float nearD = 0.0f, farD = 0.0f;
        bool leafHit = false;
        if (mine && e.x >= 0)
        {
            float4 a, b, c;
            int4 l;
            load_node(sc.nodes, e.x, a, b, c, l);
            float e0, e1;
            bool h0, h1;
            if (ray.finite)
            {
                h0 = slab_finite(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab_finite(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
            else
            {
                h0 = slab(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
                if (CULL)
                {
                    // a NaN entry (see wide_node_step) says nothing of the
                    // boxes around it, whose entries a walk may have skipped
                    e0 = fmaxf(e0, __int_as_float(e.y));
                    e1 = fmaxf(e1, __int_as_float(e.y));
                }
            }
            if (CULL)
            {
                h0 = h0 && !(e0 > cull);
                h1 = h1 && !(e1 > cull);
            }
            const bool swap = !ANY_HIT && e1 < e0;
            hNear = swap ? h1 : h0;
            hFar = swap ? h0 : h1;
            nearC = swap ? l.y : l.x;
            farC = swap ? l.x : l.y;
            nearD = swap ? e1 : e0;
            farD = swap ? e0 : e1;
        }
        else if (mine)
        {
            const int leaf = ~e.x;
            const int start = leaf >> kLeafCountBits;
            const int n = leaf & ((1 << kLeafCountBits) - 1);
            // two triangles fetched per step, as in traverse()
            for (int i = 0; i < n; i += 2)
            {
                if (ANY_HIT && found && start + i >= hit.slot)
                    break;  // a smaller slot already occludes
                float4 f[2][3];
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + start + min(i + k, n - 1));
                    f[k][0] = __ldg(tp + 0);
                    f[k][1] = __ldg(tp + 1);
                    f[k][2] = __ldg(tp + 2);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    const int slot = start + i + k;
                    const float4 ta = f[k][0], tb = f[k][1], tc = f[k][2];
                    float t, u, v;
                    if (i + k >= n || slot == skip || (ANY_HIT && found && slot >= hit.slot) ||
                        (ANY_HIT && (__float_as_uint(tc.y) & kMetaNonShadowing)) ||
                        !tri_hit(ray, v3(ta.x, ta.y, ta.z), v3(ta.w, tb.x, tb.y), v3(tb.z, tb.w, tc.x), t, u, v))
                        continue;
                    if (!ANY_HIT && ORDER == ORDER_REF && !(t == t))
                        odd = true;
                    if (ANY_HIT || t < hit.t || (t == hit.t && slot > hit.slot))
                    {
                        hit.slot = slot;
                        hit.t = t;
                        hit.u = u;
                        hit.v = v;
                        he = __int_as_float(e.y);
                        found = true;
                    }
                }
            }
            leafHit = CULL && found;
        }
        // far children first, the near ones above them
        const unsigned mFar = (__ballot_sync(kAll, hFar) >> shift) & gmask;
        const unsigned mNear = (__ballot_sync(kAll, hNear) >> shift) & gmask;
        if (hFar)
            stack[count + __popc(mFar & below)] = make_int2(farC, __float_as_int(farD));
        if (hNear)
            stack[count + __popc(mFar) + __popc(mNear & below)] = make_int2(nearC, __float_as_int(nearD));
        count += __popc(mFar) + __popc(mNear);
        if (CULL && __ballot_sync(kAll, leafHit))
        {
            float tb = hit.t;
            for (unsigned o = 1; o < G; o <<= 1)
                tb = fminf(tb, __shfl_xor_sync(kAll, tb, o));
            cull = tb * kTieCull;
        }
        __syncwarp();
    }
    for (unsigned o = 1; o < G; o <<= 1)
    {
        HitF h2;
        const bool f2 = __shfl_xor_sync(kAll, int(found), o) != 0;
        h2.slot = __shfl_xor_sync(kAll, hit.slot, o);
        h2.t = __shfl_xor_sync(kAll, hit.t, o);
        h2.u = __shfl_xor_sync(kAll, hit.u, o);
        h2.v = __shfl_xor_sync(kAll, hit.v, o);
        const float he2 = CULL ? __shfl_xor_sync(kAll, he, o) : 0.0f;
        const bool better = ANY_HIT ? h2.slot < hit.slot : (h2.t < hit.t || (h2.t == hit.t && h2.slot > hit.slot));
        if (f2 && (!found || better))
        {
            hit.slot = h2.slot;
            hit.t = h2.t;
            hit.u = h2.u;
            hit.v = h2.v;
            he = he2;
            found = true;
        }
    }
    if (!ANY_HIT)
    {
        const unsigned again = __ballot_sync(kAll, CULL ? found && he > hit.t : odd);
        if (again)
        {
            if (gl == 0 && ((again >> shift) & gmask))
                found = traverse_alone<ORDER>(sc, ray, hit, skip);
            __syncwarp();
            found = __shfl_sync(kAll, int(found), int(shift)) != 0;
            hit.slot = __shfl_sync(kAll, hit.slot, int(shift));
            hit.t = __shfl_sync(kAll, hit.t, int(shift));
            hit.u = __shfl_sync(kAll, hit.u, int(shift));
            hit.v = __shfl_sync(kAll, hit.v, int(shift));
        }
    }
    return found;
}

// Shared-memory stack entries of a warp's groups together (4 KB).
constexpr int kGroupEntries = 512;

// Ray in an instance's object space: o' = A o + b, d' = A d. d' is not
// renormalised, so a hit's parameter t is the same in both spaces and the
// levels share one closest distance. (The reference's Instance normalises
// the direction and recomputes the world distance from the transformed hit
// point, Instance.cpp:65-100: the same t in exact arithmetic.)
__device__ __forceinline__ RayF instance_ray(const DevInstance& in, const RayF& r)
{
    if (in.identity)
        return r;
    V3 o = v3(__fmaf_rn(in.r0.x, r.o.x, __fmaf_rn(in.r0.y, r.o.y, __fmaf_rn(in.r0.z, r.o.z, in.r0.w))),
              __fmaf_rn(in.r1.x, r.o.x, __fmaf_rn(in.r1.y, r.o.y, __fmaf_rn(in.r1.z, r.o.z, in.r1.w))),
              __fmaf_rn(in.r2.x, r.o.x, __fmaf_rn(in.r2.y, r.o.y, __fmaf_rn(in.r2.z, r.o.z, in.r2.w))));
    V3 d = v3(__fmaf_rn(in.r0.x, r.d.x, __fmaf_rn(in.r0.y, r.d.y, __fmul_rn(in.r0.z, r.d.z))),
              __fmaf_rn(in.r1.x, r.d.x, __fmaf_rn(in.r1.y, r.d.y, __fmul_rn(in.r1.z, r.d.z))),
              __fmaf_rn(in.r2.x, r.d.x, __fmaf_rn(in.r2.y, r.d.y, __fmul_rn(in.r2.z, r.d.z))));
    return make_ray(o, d, r.tmin, r.tmax);
}

__device__ __forceinline__ DevInstance load_instance(const DevInstance* __restrict__ p, int k)
{
    const float4* q = reinterpret_cast<const float4*>(p + k);
    DevInstance in;
    in.r0 = __ldg(q + 0);
    in.r1 = __ldg(q + 1);
    in.r2 = __ldg(q + 2);
    const int4 m = __ldg(reinterpret_cast<const int4*>(q + 3));
    in.rootLink = m.x;
    in.material = m.y;
    in.primBase = m.z;
    in.identity = m.w;
    return in;
}

// Two-level traversal: the top-level BVH over instances (nearest child
// first, culled by the closest hit), and inside each instance its mesh's
// BVH with the object-space ray. `skip` / `skipInst` name the triangle (and
// its instance) a secondary ray leaves from. Instance materials that are
// nonShadowing are skipped by any-hit queries (Instance.cpp:25-26).
template <bool ANY_HIT, bool COUNT>
__device__ __noinline__ bool traverse_instanced(const DevScene& sc, const RayF& ray, HitF& hit, TravCount& cnt,
                                                int& err, int skip, int skipInst)
{
    constexpr int kTopStack = 32;
    int stack[kTopStack];
    float sdist[kTopStack];
    int sp = 0;
    int cur = sc.tlasRoot;
    bool found = false;
    DevScene mesh = sc;
    while (true)
    {
        if (cur >= 0)
        {
            float4 a, b, c;
            int4 l;
            load_node(sc.tlas, cur, a, b, c, l);
            float e0, e1;
            bool h0, h1;
            if (ray.finite)
            {
                h0 = slab_finite(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab_finite(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
            else
            {
                h0 = slab(ray, a.x, a.y, a.z, a.w, c.x, c.y, e0);
                h1 = slab(ray, b.x, b.y, b.z, b.w, c.z, c.w, e1);
            }
            if (!ANY_HIT)
            {
                h0 = h0 && !(e0 > hit.t);
                h1 = h1 && !(e1 > hit.t);
            }
            if (h0 && h1)
            {
                int nearC = l.x, farC = l.y;
                float farD = e1;
                if (!ANY_HIT && e1 < e0)
                {
                    nearC = l.y;
                    farC = l.x;
                    farD = e0;
                }
                if (sp >= kTopStack)
                {
                    err = 1;
                    return found;
                }
                stack[sp] = farC;
                sdist[sp] = farD;
                sp++;
                cur = nearC;
                continue;
            }
            if (h0)
            {
                cur = l.x;
                continue;
            }
            if (h1)
            {
                cur = l.y;
                continue;
            }
        }
        else
        {
            const int leaf = ~cur;
            const int start = leaf >> kLeafCountBits;
            const int count = leaf & ((1 << kLeafCountBits) - 1);
            for (int i = 0; i < count; ++i)
            {
                const int k = start + i;
                const DevInstance in = load_instance(sc.instances, k);
                if (ANY_HIT && in.material >= 0 &&
                    (__float_as_uint(__ldg(&sc.mats[in.material].emittance.w)) & kMatNonShadowing))
                    continue;
                const RayF r2 = instance_ray(in, ray);
                mesh.rootLink = in.rootLink;
                HitF h2 = hit;
                if (traverse<ANY_HIT, ORDER_NEAREST, COUNT>(mesh, r2, h2, cnt, err, k == skipInst ? skip : -1))
                {
                    hit = h2;
                    hit.inst = k;
                    found = true;
                    if (ANY_HIT)
                        return true;
                }
            }
        }
        while (true)
        {
            if (sp == 0)
                return found;
            sp--;
            cur = stack[sp];
            if (!ANY_HIT && sdist[sp] > hit.t)
                continue;
            break;
        }
    }
}

// Either traversal, by the scene's kind.
template <bool ANY_HIT, int ORDER, bool COUNT>
__device__ __forceinline__ bool traverse_scene(const DevScene& sc, const RayF& ray, HitF& hit, TravCount& cnt,
                                               int& err, int skip, int skipInst)
{
    if (sc.numInstances > 0)
        return traverse_instanced<ANY_HIT, COUNT>(sc, ray, hit, cnt, err, skip, skipInst);
    return traverse<ANY_HIT, ORDER, COUNT>(sc, ray, hit, cnt, err, skip);
}

}  // namespace rcx
