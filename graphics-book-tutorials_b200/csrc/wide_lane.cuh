// The ordered traversal's call into the preorder steps, shared by its kernels.
#pragma once
#include "wide_bvh.cuh"

namespace wfb {
namespace {

// The preorder steps, as a call: the few rays the ordered traversal does not answer (wide_bvh.cuh). Returns
// {t, prim bits}.
__device__ __noinline__ float2 exact_trace(const float4* nodes, int n_nodes, const float4* prims, int n_spheres,
                                           float ox, float oy, float oz, float dx, float dy, float dz, float tmax,
                                           int anyhit) {
    wf::HitRecord h;
    exact_trace_body(nodes, n_nodes, prims, n_spheres, wf::Vec3{ox, oy, oz}, wf::Vec3{dx, dy, dz}, tmax, anyhit != 0, &h);
    return make_float2(h.t, __int_as_float(h.prim));
}

}  // namespace
}  // namespace wfb
