// Collapse of the preorder skip-link BVH into wide nodes, shared by the device build (wide_build.cu)
// and the host check (trav_check.cu). `nodes` are packed records (dev_scene.cuh).
#pragma once
#include "wide_bvh.cuh"

namespace wfb {

#if defined(__CUDACC__)

WF_HD float i2f_bits(int i) {
#if defined(__CUDA_ARCH__)
    return __int_as_float(i);
#else
    float f;
    __builtin_memcpy(&f, &i, 4);
    return f;
#endif
}

WF_HD int subtree_end(const float4* nodes, int nn, int i) {
    const int skip = f2i(nodes[2 * i].w);
    return skip < 0 ? nn : skip;
}

// Up to 4 children under construction, indexed through unrolled selects so that they stay in registers (in local
// memory the walk of a level took 20 us).
struct WideKids {
    int id[kWideArity];
    float area[kWideArity];  // surface, -1 for a leaf or a node not to be opened
    int n;
};
WF_HD void put_kid(WideKids& k, int at, int id, float area) {
#pragma unroll
    for (int j = 0; j < kWideArity; ++j)
        if (j == at) {
            k.id[j] = id;
            k.area[j] = area;
        }
}
// Preorder node c as child `at`; returns the end of its subtree.
WF_HD int load_kid(const float4* nodes, int nn, int c, WideKids& k, int at) {
    const float4 lo = nodes[2 * c], hi = nodes[2 * c + 1];
    const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
    put_kid(k, at, c, f2i(hi.w) >= 0 ? -1.0f : x * y + y * z + z * x);
    return f2i(lo.w) < 0 ? nn : f2i(lo.w);
}

// The preorder nodes that become the children of the wide node standing for `root`: its direct children (root + 1, then
// the end of each one's subtree, up to root's own end), then, while there is room, the internal one with the
// largest surface is replaced by its own children (the box most often entered is the one worth opening). A root that is
// a leaf is its own only child. False for a node with no children or more than 4.
WF_HD bool wide_children(const float4* nodes, int nn, int root, WideKids* out) {
    WideKids k;
#pragma unroll
    for (int j = 0; j < kWideArity; ++j) {
        k.id[j] = 0;
        k.area[j] = -1.0f;
    }
    k.n = 0;
    if (f2i(nodes[2 * root + 1].w) >= 0) {
        load_kid(nodes, nn, root, k, k.n++);
        *out = k;
        return true;
    }
    for (int c = root + 1, end = subtree_end(nodes, nn, root); c < end;) {
        if (k.n == kWideArity) return false;
        c = load_kid(nodes, nn, c, k, k.n++);
    }
    while (k.n > 0) {
        int best = -1, id = 0;
        float best_area = -1.0f;
#pragma unroll
        for (int j = 0; j < kWideArity; ++j)
            if (j < k.n && k.area[j] > best_area) {
                best = j;
                best_area = k.area[j];
                id = k.id[j];
            }
        if (best < 0) break;
        const int end = subtree_end(nodes, nn, id);
        int m = 0;
        for (int c = id + 1; c < end && m <= kWideArity; ++m) c = subtree_end(nodes, nn, c);
        if (m == 0 || m > kWideArity) return false;
        if (k.n - 1 + m > kWideArity) {
            put_kid(k, best, id, -1.0f);
            continue;
        }
        int c = load_kid(nodes, nn, id + 1, k, best);
        while (c < end) c = load_kid(nodes, nn, c, k, k.n++);
    }
    *out = k;
    return k.n > 0;
}

// Writes the wide node: the grid covers the children's boxes with a margin at both ends, and each plane is
// the nearest grid plane outside the box plane by kPlaneMargin steps or more (less the rounding of the position in steps,
// 255 * 2^-22 of one, which is far below the margin). codes[] as in the node layout.
WF_HD void wide_write(const float4* nodes, const WideKids& kids, const int (&codes)[kWideArity], float4* out) {
    const int k = kids.n;
    unsigned lo_q[3] = {~0u, ~0u, ~0u}, hi_q[3] = {0u, 0u, 0u};  // unused slots: inside out
    float origin[3], step[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        auto at = [&](const float4& v) { return x == 0 ? v.x : x == 1 ? v.y : v.z; };
        float lo = INFINITY, hi = -INFINITY;
        float box_lo[kWideArity], box_hi[kWideArity];
#pragma unroll
        for (int i = 0; i < kWideArity; ++i) {
            box_lo[i] = box_hi[i] = 0.0f;
            if (i < k) {
                box_lo[i] = at(nodes[2 * kids.id[i]]);
                box_hi[i] = at(nodes[2 * kids.id[i] + 1]);
                lo = fminf(lo, box_lo[i]);
                hi = fmaxf(hi, box_hi[i]);
            }
        }
        if (k == 0) lo = hi = 0.0f;
        // The origin lies below lo, and 255 steps reach beyond hi, by more than the margin: the step is at least 8
        // roundings of a coordinate (size * 2^-24), so that the origin's own rounding is well below a step; it never vanishes.
        const float size = fmaxf(fabsf(lo), fabsf(hi));
        const float s = fmaxf(fmaxf((hi - lo) * (1.0f / 254.0f), size * 4.8e-7f), 1e-11f) * 1.000001f;
        step[x] = s;
        origin[x] = lo - 0.25f * s;
        const float per_step = 1.0f / s;
#pragma unroll
        for (int i = 0; i < kWideArity; ++i) {
            if (i >= k) continue;
            const float a = (box_lo[i] - origin[x]) * per_step - kPlaneMargin;
            const float b = (box_hi[i] - origin[x]) * per_step + kPlaneMargin;
            const unsigned qa = (unsigned)fminf(fmaxf(floorf(a), 0.0f), 255.0f);
            const unsigned qb = (unsigned)fminf(fmaxf(ceilf(b), 0.0f), 255.0f);
            lo_q[x] = (lo_q[x] & ~(255u << (8 * i))) | (qa << (8 * i));
            hi_q[x] = (hi_q[x] & ~(255u << (8 * i))) | (qb << (8 * i));
        }
    }
    auto bits = [](unsigned u) { return i2f_bits((int)u); };
    out[0] = make_float4(origin[0], origin[1], step[0] * 32768.0f, step[1] * 32768.0f);
    out[1] = make_float4(origin[2], step[2] * 32768.0f, bits(lo_q[0]), bits(hi_q[0]));
    out[2] = make_float4(bits(lo_q[1]), bits(hi_q[1]), bits(lo_q[2]), bits(hi_q[2]));
    out[3] = make_float4(i2f_bits(codes[0]), i2f_bits(codes[1]), i2f_bits(codes[2]), i2f_bits(codes[3]));
}

// One primitive record lies inside the leaf box [lo, hi] up to a few ulp of the coordinates (its far vertices
// are p0 + e, each a rounded difference).
WF_HD bool prim_in_box(const float4* rec, int n_spheres, const float4& lo, const float4& hi) {
    auto inside = [&](float x, float y, float z, float r) {
        const float tx = 4.8e-7f * (fabsf(x) + r), ty = 4.8e-7f * (fabsf(y) + r), tz = 4.8e-7f * (fabsf(z) + r);
        return x - r >= lo.x - tx && x + r <= hi.x + tx && y - r >= lo.y - ty && y + r <= hi.y + ty &&
               z - r >= lo.z - tz && z + r <= hi.z + tz;
    };
    const float4 p = rec[0], a = rec[1], b = rec[2];
    if (f2i(p.w) < n_spheres) return a.x >= 0.0f && inside(p.x, p.y, p.z, a.x);
    // the sum p0 + e is off by an ulp of the larger of p0 and the vertex
    auto vertex = [&](float x, float y, float z) {
        const float vx = p.x + x, vy = p.y + y, vz = p.z + z;
        const float tx = 4.8e-7f * (fabsf(p.x) + fabsf(x)), ty = 4.8e-7f * (fabsf(p.y) + fabsf(y)),
                    tz = 4.8e-7f * (fabsf(p.z) + fabsf(z));
        return vx >= lo.x - tx && vx <= hi.x + tx && vy >= lo.y - ty && vy <= hi.y + ty && vz >= lo.z - tz &&
               vz <= hi.z + tz;
    };
    return inside(p.x, p.y, p.z, 0.0f) && vertex(a.x, a.y, a.z) && vertex(b.x, b.y, b.z);
}

WF_HD bool box_in_range(const float4& lo, const float4& hi) {
    return fabsf(lo.x) < kCoordMax && fabsf(lo.y) < kCoordMax && fabsf(lo.z) < kCoordMax && fabsf(hi.x) < kCoordMax &&
           fabsf(hi.y) < kCoordMax && fabsf(hi.z) < kCoordMax;
}

#endif  // __CUDACC__

}  // namespace wfb
