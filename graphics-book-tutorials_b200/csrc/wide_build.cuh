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

// Direct children of internal node i: i + 1, then the end of each child's subtree, up to i's own end.
// Returns their number, kWideArity + 1 when there are more than fit.
WF_HD int direct_children(const float4* nodes, int nn, int i, int* out) {
    int k = 0;
    for (int c = i + 1, end = subtree_end(nodes, nn, i); c < end; c = subtree_end(nodes, nn, c)) {
        if (k == kWideArity) return k + 1;
        out[k++] = c;
    }
    return k;
}

// The preorder nodes that become the children of the wide node standing for `root`: its direct
// children, then, while there is room, the internal one with the largest surface is replaced by its own
// children (the box most often entered is the one worth opening). A root that is a leaf is its own only child. Returns
// their number, -1 for a node with too many children.
WF_HD int wide_children(const float4* nodes, int nn, int root, int* kids) {
    if (f2i(nodes[2 * root + 1].w) >= 0) {
        kids[0] = root;
        return 1;
    }
    int k = direct_children(nodes, nn, root, kids);
    if (k > kWideArity || k == 0) return -1;
    bool tried[kWideArity] = {};
    for (;;) {
        int best = -1;
        float best_area = -1.0f;
        for (int i = 0; i < k; ++i) {
            const float4 lo = nodes[2 * kids[i]], hi = nodes[2 * kids[i] + 1];
            if (f2i(hi.w) >= 0 || tried[i]) continue;
            const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
            const float area = x * y + y * z + z * x;
            if (area > best_area) {
                best_area = area;
                best = i;
            }
        }
        if (best < 0) return k;
        int sub[kWideArity];
        const int m = direct_children(nodes, nn, kids[best], sub);
        if (m > kWideArity || m == 0) return -1;
        if (k - 1 + m > kWideArity) {
            tried[best] = true;
            continue;
        }
        kids[best] = sub[0];
        for (int j = 1; j < m; ++j) kids[k++] = sub[j];
    }
}

// Writes the wide node: the grid covers the children's boxes with a margin at both ends, and each plane is
// the nearest grid plane outside the box plane by kPlaneMargin steps or more. In doubles, so that the margin is exact
// to far below itself; codes[] as in the node layout.
WF_HD void wide_write(const float4* nodes, const int* kids, const int* codes, int k, float4* out) {
    unsigned lo_q[3] = {~0u, ~0u, ~0u}, hi_q[3] = {0u, 0u, 0u};  // unused slots: inside out
    float origin[3], step[3];
    for (int x = 0; x < 3; ++x) {
        auto at = [&](const float4& v) { return x == 0 ? v.x : x == 1 ? v.y : v.z; };
        float lo = INFINITY, hi = -INFINITY;
        for (int i = 0; i < k; ++i) {
            lo = fminf(lo, at(nodes[2 * kids[i]]));
            hi = fmaxf(hi, at(nodes[2 * kids[i] + 1]));
        }
        if (k == 0) lo = hi = 0.0f;
        // The origin lies below lo, and 255 steps reach beyond hi, by more than the margin; the step is
        // large enough that the origin's rounding (an ulp of its size) is well below it, and never vanishes.
        const double extent = (double)hi - (double)lo;
        const double size = fmax(fabs((double)lo), fabs((double)hi));
        const double s = fmax(fmax(extent / 254.0, size * 4.8e-7), 1e-11);
        step[x] = (float)(s * 1.0000002);
        origin[x] = (float)((double)lo - 0.25 * s);
        const double per_step = 1.0 / (double)step[x];
        for (int i = 0; i < k; ++i) {
            const double a = ((double)at(nodes[2 * kids[i]]) - (double)origin[x]) * per_step - kPlaneMargin;
            const double b = ((double)at(nodes[2 * kids[i] + 1]) - (double)origin[x]) * per_step + kPlaneMargin;
            const unsigned qa = (unsigned)fmin(fmax(floor(a), 0.0), 255.0);
            const unsigned qb = (unsigned)fmin(fmax(ceil(b), 0.0), 255.0);
            lo_q[x] = (lo_q[x] & ~(255u << (8 * i))) | (qa << (8 * i));
            hi_q[x] = (hi_q[x] & ~(255u << (8 * i))) | (qb << (8 * i));
        }
    }
    auto bits = [](unsigned u) { return i2f_bits((int)u); };
    out[0] = make_float4(origin[0], origin[1], step[0] * 32768.0f, step[1] * 32768.0f);
    out[1] = make_float4(origin[2], step[2] * 32768.0f, bits(lo_q[0]), bits(hi_q[0]));
    out[2] = make_float4(bits(lo_q[1]), bits(hi_q[1]), bits(lo_q[2]), bits(hi_q[2]));
    int c[kWideArity];
    for (int i = 0; i < kWideArity; ++i) c[i] = i < k ? codes[i] : 0;
    out[3] = make_float4(i2f_bits(c[0]), i2f_bits(c[1]), i2f_bits(c[2]), i2f_bits(c[3]));
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
