// Ordered traversal of a 4-wide tree over the leaves of the scene's preorder BVH.
//
// Preorder traversal (dev_scene.cuh, box_step) visits a node's children in a fixed order, so a
// closest-hit ray that reaches the far child first tests most of what lies behind its hit: on
// icospheres 92.5 box steps and 6.7 primitive tests per ray, against 16.0 wide nodes and 3.2 primitive
// tests when the nearest child goes first. The hit must still be the one preorder traversal returns
// (a primitive replaces the best only when strictly nearer, and a leaf is entered only when its box
// test passes against the tmax of that moment). What that leaves open is only rounding:
//
//  * Let m be the smallest t of all primitive hits in leaves whose box the ray meets, and let it be
//    reached by one primitive alone: every other hit is farther than m * kTieUp. When that
//    primitive's leaf box is entered no later than m * kEntryUp, preorder traversal reaches the leaf
//    with a tmax beyond that entry (any hit it holds by then is farther), enters it and takes the hit;
//    nothing replaces it. So the ordered traversal returns the same primitive, with the same t, for
//    it runs the same primitive test.
//  * Two hits within kTieUp of each other at the end (a shared edge, coincident surfaces), a best
//    hit whose leaf box is missed or entered late, a ray whose 1/d is not finite or beyond kInvMax,
//    and a full stack all send the ray through the preorder steps instead (exact_trace).
//  * A subtree is skipped only when its box is entered beyond kCullSlack times the best hit. A primitive in there is
//    nearer than the best only if the t it reports lies in front of its own leaf's box by more than that factor. This is the
//    one case in which the two traversals' hits differ: preorder traversal may then return that primitive, whose t is
//    wrong, the ordered one the nearest of the others. It takes a triangle test with a determinant at the level of its
//    rounding, that is a ray within about 1e-4 of the plane of a triangle that it still meets (or a sliver), and
//    another surface in the gap. Of 10^6 rays aimed to graze a smooth mesh of well-shaped triangles at 1e-3 / 1e-4 / 1e-5
//    rad, 1 / 24 / 179 differ; of 300,000 through slivers of width 1e-5, 1; of 494,194 rays of real paths, none. A slack of
//    1/128 leaves 1 / 4 / 58 for 1% more nodes, one of 1/16 0 / 0 / 13 for 11%: no slack closes it. Renders
//    with speculation off take the plain preorder steps and have no such case.
//  * Any-hit queries (shadow rays) have a fixed tmax, so whether a leaf is entered depends on its
//    box alone: occluded when some leaf whose box passes holds a primitive hit below tmax, in any
//    order. Exact, with the leaf's own box test run on the hit that ended the query (should it fail, the
//    preorder steps answer).
//
// Conditions on the tree, checked at upload (wide_build.cu): nested boxes, every primitive inside
// its leaf's box, each prim_order entry in one leaf, finite coordinates below kCoordMax, at most 4
// children per node. A tree that fails one keeps the preorder traversal.
//
// Box tests of internal nodes are conservative instead of exact: the planes are stored in 8 bits, rounded outwards
// with a margin (kPlaneMargin steps) that covers the rounding of the slab distances below, and the interval is
// compared with a relative margin (kBoxSlack) that covers the exact test's own two roundings. So a box that passes the
// exact test always passes here.
#pragma once
#include "dev_scene.cuh"

namespace wfb {

constexpr float kCullSlack = 1.0f + 1.0f / 1024.0f;   // subtrees are skipped beyond best * this
constexpr float kTieUp = 1.0f + 1.0f / 262144.0f;     // hits within these factors of the best are ties
constexpr float kTieDown = 1.0f - 1.0f / 262144.0f;
constexpr float kEntryUp = 1.0f + 1.0f / 524288.0f;   // the best hit's leaf box is entered by best * this
constexpr float kBoxSlack = 1.0f + 1.0f / 1048576.0f;
constexpr float kInvMax = 1.099511627776e12f;    // 2^40, as for coordinates: no overflow in (plane - o) / d
constexpr float kCoordMax = 1.099511627776e12f;

// A wide node is 4 float4 (64 B, two 32-byte loads): a grid (origin, step per axis) and the planes of up to 4 child
// boxes on it, 8 bits each (after Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
// BVHs", HPG 2017, whose nodes have 8 children), child k's in byte k:
//   {origin.x, origin.y, step.x, step.y} {origin.z, step.z, lo.x[4], hi.x[4]}
//   {lo.y[4], hi.y[4], lo.z[4], hi.z[4]} {code}[4]
// (the steps stored times 2^15, see plane_of)
// code: > 0 a leaf (its leaf encoding, start * 16 + count), < 0 ~(wide node index). A slot without a child has inside-out
// planes and the code of the empty leaf (empty_leaf): seen from so far that the whole node is shorter than the box test's
// margin, inside-out planes are met like any others, and a code that is no node would end the walk there. The check for it
// in wide_node_step instead cost 1.2% on the heightfield and 2% in the wavefront on icospheres (1280x720).
// A plane q lies at origin + q * step. Icospheres: 80K nodes, 5.1 MB, where the preorder nodes are 10.4 MB.
constexpr int kWideFloat4 = 4;
constexpr int kWideArity = 4;
constexpr int kWideMaxLevels = 96;  // a deeper wide tree keeps the preorder traversal
constexpr float kPlaneMargin = 1.0f / 64.0f;

// The empty leaf: one record behind the scene's n, a triangle without edges, which no ray hits (its determinant is 0).
WF_HD int empty_leaf(int n) { return (n << kLeafCountBits) | 1; }
constexpr long long kMaxWidePrims = kMaxLeafStart;  // primitive entries, so that its code is a leaf's

// Stack entries per lane kept in shared memory; deeper ones go to the lane's local memory (on icospheres 1 ray in 6,000
// holds more than 15, none more than 18).
constexpr int kStackShared = 16;
constexpr int kStackLocal = 32;

#if defined(__CUDACC__)

// 1/d finite, not NaN and within the range where plane * (1/d) neither overflows nor vanishes.
WF_HD bool wide_ray(const TravRay& ray) {
    const float x = fabsf(ray.inv_d.x), y = fabsf(ray.inv_d.y), z = fabsf(ray.inv_d.z);
    return x < kInvMax && y < kInvMax && z < kInvMax && fminf(fminf(x, y), z) > 1.0f / kInvMax;
}

// Lane state of the ordered traversal. `cur`: the next node (< 0 wide node, > 0 leaf waiting while
// another is pending, 0 none); `pend`: the leaf being tested (box_step's encoding); `best`: the current
// tmax; `rank`: prim_order position of the best hit, -1 none; `redo` nonzero: the ray goes to exact_trace
// (kRedoTie: another hit as near as the best one; kRedoRay: the ray itself is not for this traversal).
enum : int { kRedoTie = 1, kRedoRay = 2 };
struct WideState {
    int cur, pend;
    int sp, base;  // stack position, and where it is empty (both in the stack's own units)
    int rank;
    float best;
    int redo;
};

WF_HD void wide_begin(wf::Vec3 d, float tmax, bool has_nodes, int stack_base, TravRay* ray, WideState* s) {
    ray->d = d;
    ray->inv_d = wf::Vec3{1.0f / d.x, 1.0f / d.y, 1.0f / d.z};
    const bool fit = wide_ray(*ray);
    s->cur = has_nodes && fit ? ~0 : 0;
    s->pend = 0;
    s->sp = s->base = stack_base;
    s->rank = -1;
    s->best = tmax;
    s->redo = fit ? 0 : kRedoRay;
}

// A lane's stack of nodes, one column per thread, so that lanes at different depths never meet in a bank: the first
// entries in shared memory (WideState::sp is the word index there), deeper ones in local memory.
template <int BLOCK>
struct LaneStack {
    int* words;  // kStackShared * BLOCK words, shared
    int* deep;   // kStackLocal words, local
    WF_HD void push3(WideState& s, int a, bool pa, int b, bool pb, int c, bool pc) {
        if (s.sp < (kStackShared - 2) * BLOCK) {  // room for three
            if (pa) { words[s.sp] = a; s.sp += BLOCK; }
            if (pb) { words[s.sp] = b; s.sp += BLOCK; }
            if (pc) { words[s.sp] = c; s.sp += BLOCK; }
        } else {
            if (pa) push_deep(s, a);
            if (pb) push_deep(s, b);
            if (pc) push_deep(s, c);
        }
    }
    WF_HD void push_deep(WideState& s, int code) {
        if (s.sp < kStackShared * BLOCK) words[s.sp] = code;
        else if (s.sp < (kStackShared + kStackLocal) * BLOCK) deep[(s.sp - s.base) / BLOCK - kStackShared] = code;
        else {
            s.redo |= kRedoRay;
            return;
        }
        s.sp += BLOCK;
    }
    WF_HD void pop(WideState& s) const {
        if (s.sp == s.base) return;
        s.sp -= BLOCK;
        s.cur = s.sp < kStackShared * BLOCK ? words[s.sp] : deep[(s.sp - s.base) / BLOCK - kStackShared];
    }
};

// The lane's next node: `cur` stays while it is usable; a leaf becomes the pending one when none is; an
// empty `cur` is refilled from the stack.
#pragma nv_exec_check_disable
template <class Stack>
WF_HD void wide_next(WideState& s, Stack& stack) {
    if (s.cur == 0) stack.pop(s);
    if (s.cur > 0 && s.pend == 0) {
        s.pend = s.cur;
        s.cur = 0;
        stack.pop(s);
    }
}

// 1 + q * 2^-15 for the byte q of child k: one byte permute.
template <int K>
WF_HD float plane_of(unsigned bytes) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(__byte_perm(bytes, 0x3f800000u, 0x7604u | (K << 4)));
#else
    const unsigned q = (bytes >> (8 * K)) & 255u;
    const unsigned u = 0x3f800000u | (q << 8);
    float f;
    __builtin_memcpy(&f, &u, 4);
    return f;
#endif
}

// {a.x * b.x + c.x, a.y * b.y + c.y}: one packed instruction on the device.
WF_HD float2 fma2(float2 a, float2 b, float2 c) {
#if defined(__CUDA_ARCH__)
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}

WF_HD unsigned f2u(float f) { return (unsigned)f2i(f); }

// A ray against a node's grid: with a = step / d and b = (origin - o) / d, plane q is met at q a + b = (1 + q 2^-15)
// (2^15 a) + (b - 2^15 a), whose rounding error is below 2^-22 of the distance plus 0.0021 of a step. Plane bytes are
// chosen by the direction's sign.
struct WideGrid {
    unsigned near_x, near_y, near_z, far_x, far_y, far_z;
    float2 a_xy, b_xy, a_zz, b_zz;
    float limit;
};

// Entry distance of child K's box, infinite when the box is missed.
template <int K>
WF_HD float child_entry(const WideGrid& g) {
    const float2 n = fma2(make_float2(plane_of<K>(g.near_x), plane_of<K>(g.near_y)), g.a_xy, g.b_xy);
    const float2 f = fma2(make_float2(plane_of<K>(g.far_x), plane_of<K>(g.far_y)), g.a_xy, g.b_xy);
    const float2 z = fma2(make_float2(plane_of<K>(g.near_z), plane_of<K>(g.far_z)), g.a_zz, g.b_zz);
    const float t0 = fmaxf(fmaxf(n.x, n.y), fmaxf(z.x, wf::kRayEps));
    const float t1 = fminf(fminf(f.x, f.y), fminf(z.y, g.limit));
    return t0 <= t1 * kBoxSlack ? t0 : INFINITY;
}

// The lane's wide node: its children are tested together; the nearest one that is met becomes `cur`, the others go
// on the stack. Neither a full sort nor entry distances on the stack (to drop entries behind a nearer
// hit when they come up) pay: they save 1% and 5-12% of the nodes.
#pragma nv_exec_check_disable
template <class Stack>
WF_HD void wide_node_step(const float4* __restrict__ wide, const wf::Vec3& o, const wf::Vec3& inv, WideState& s,
                          Stack& stack) {
    const float4* n = wide + (size_t)kWideFloat4 * (unsigned)~s.cur;
    float4 q0, q1, q2, q3;
#if defined(__CUDA_ARCH__)
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(q0.x), "=f"(q0.y), "=f"(q0.z), "=f"(q0.w), "=f"(q1.x), "=f"(q1.y), "=f"(q1.z), "=f"(q1.w)
        : "l"(n));
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(q2.x), "=f"(q2.y), "=f"(q2.z), "=f"(q2.w), "=f"(q3.x), "=f"(q3.y), "=f"(q3.z), "=f"(q3.w)
        : "l"(n + 2));
#else
    q0 = n[0];
    q1 = n[1];
    q2 = n[2];
    q3 = n[3];
#endif
    const bool sx = inv.x < 0.0f, sy = inv.y < 0.0f, sz = inv.z < 0.0f;
    WideGrid g;
    g.near_x = f2u(sx ? q1.w : q1.z);
    g.far_x = f2u(sx ? q1.z : q1.w);
    g.near_y = f2u(sy ? q2.y : q2.x);
    g.far_y = f2u(sy ? q2.x : q2.y);
    g.near_z = f2u(sz ? q2.w : q2.z);
    g.far_z = f2u(sz ? q2.z : q2.w);
    g.a_xy = make_float2(q0.z * inv.x, q0.w * inv.y);
    g.b_xy = fma2(make_float2(q0.x - o.x, q0.y - o.y), make_float2(inv.x, inv.y), make_float2(-g.a_xy.x, -g.a_xy.y));
    const float az = q1.y * inv.z, bz = fmaf(q1.x - o.z, inv.z, -az);
    g.a_zz = make_float2(az, az);
    g.b_zz = make_float2(bz, bz);
    g.limit = s.best * kCullSlack;
    // insertion: the nearer of the current choice and the next child stays, the other goes on the stack
    float tc = child_entry<0>(g);
    int cur = f2i(q3.x);
    auto next = [&](float t, int code, int& out) {
        const bool nearer = t < tc;
        out = nearer ? cur : code;
        cur = nearer ? code : cur;
        const float behind = fmaxf(t, tc);
        tc = fminf(t, tc);
        return behind < INFINITY;
    };
    int c1, c2, c3;
    const bool p1 = next(child_entry<1>(g), f2i(q3.y), c1);
    const bool p2 = next(child_entry<2>(g), f2i(q3.z), c2);
    const bool p3 = next(child_entry<3>(g), f2i(q3.w), c3);
    s.cur = tc < INFINITY ? cur : 0;
    stack.push3(s, c1, p1, c2, p2, c3, p3);
}

// The third vector of a primitive record. It is loaded along with the first two although spheres have no use for it: left to
// the branch that uses it (where the compiler moves a plain load), it waits for the first vector to arrive.
WF_HD float4 load_e2(const float4* rec) {
#if defined(__CUDA_ARCH__)
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(rec + 2));
    return v;
#else
    return rec[2];
#endif
}

// One primitive of the pending leaf against the ray, as prim_step tests it. Closest hit: hits up to
// best * kTieUp are seen, so that a tie on either side of the best sets `redo`; a clearly nearer hit
// clears it again. Any hit: the first hit ends the query (wide_resolve runs its leaf's own box test).
WF_HD void wide_prim_step(const float4* __restrict__ prims, int n_spheres, const wf::Vec3& o, const TravRay& ray,
                          bool anyhit, WideState& s) {
    const int rank = s.pend >> kLeafCountBits;
    const float4* rec = prims + 3 * rank;
    const float4 q2 = load_e2(rec);
    const float4 q0 = ro_load(rec);
    const float4 q1 = ro_load(rec + 1);
    wf::Ray r;
    r.o = o;
    r.d = ray.d;
    r.tmin = wf::kRayEps;
    r.tmax = anyhit ? s.best : s.best * kTieUp;
    float t, u, v;
    bool hit;
    if (f2i(q0.w) < n_spheres)
        hit = wf::hit_sphere_core(wf::Vec3{q0.x, q0.y, q0.z}, q1.x, r, &t);
    else
        hit = wf::hit_triangle_core(wf::Vec3{q0.x, q0.y, q0.z}, wf::Vec3{q1.x, q1.y, q1.z},
                                    wf::Vec3{q2.x, q2.y, q2.z}, r, &t, &u, &v);
    s.pend += (1 << kLeafCountBits) - 1;
    if ((s.pend & kLeafCountMask) == 0) s.pend = 0;
    if (!hit) return;
    if (anyhit) {
        s.rank = rank;
        s.cur = 0;
        s.pend = 0;
        s.sp = s.base;
        return;
    }
    s.redo = (s.redo & ~kRedoTie) | (t >= s.best * kTieDown ? kRedoTie : 0);
    if (t < s.best) {
        s.best = t;
        s.rank = rank;
    }
}

// The preorder steps from the ray's start: what the ordered traversal hands over to.
WF_HD void exact_trace_body(const float4* __restrict__ nodes, int n_nodes, const float4* __restrict__ prims,
                            int n_spheres, const wf::Vec3& o, const wf::Vec3& d, float tmax, bool anyhit,
                            wf::HitRecord* h) {
    TravRay ray;
    int node, pend = 0;
    traversal_begin(n_nodes, d, tmax, &ray, &node, h);
    while (node >= 0 || pend != 0) {
        if (pend != 0) prim_step(prims, n_spheres, o, ray, anyhit, node, pend, *h);
        else box_step_on(ro_load(nodes + 2 * node), ro_load(nodes + 2 * node + 1), n_nodes, o, ray, h->t, node, pend);
    }
}

// A ray at its end: true when what it found is what preorder traversal finds; `h` gets it. Closest hit: the best hit
// has no tie, and its leaf's box is met, and entered by best * kEntryUp. Any hit: the leaf's box passes with the
// ray's tmax; else another leaf may hold the hit. A miss without `redo` is a miss.
WF_HD bool wide_resolve(const float4* __restrict__ prims, const float4* __restrict__ nodes, const wf::Vec3& o,
                        const TravRay& ray, bool anyhit, const WideState& s, wf::HitRecord* h) {
    h->t = s.best;
    h->prim = -1;
    if (s.rank < 0 || (s.redo && !anyhit)) return s.redo == 0;
    h->prim = f2i(ro_load(prims + 3 * s.rank).w);
    const int leaf = f2i(ro_load(prims + 3 * s.rank + 1).w) - 1;
    const float4 a = ro_load(nodes + 2 * leaf), b = ro_load(nodes + 2 * leaf + 1);
    return wf::hit_box_minmax(wf::Vec3{a.x, a.y, a.z}, wf::Vec3{b.x, b.y, b.z}, o, ray.inv_d, wf::kRayEps,
                              anyhit ? s.best : s.best * kEntryUp);
}

#endif  // __CUDACC__

}  // namespace wfb
