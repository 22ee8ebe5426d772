// Device parts of the ordered traversal (wide_bvh.cuh) that its kernels share: the lane's stack and the call into the
// preorder steps.
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

// A lane's stack of nodes, one column per thread, so that lanes at different depths never meet in a bank: the first
// entries in shared memory (WideState::sp is the word index there), deeper ones in local memory.
template <int BLOCK>
struct LaneStack {
    int* words;  // kStackShared * BLOCK words, shared
    int* deep;   // kStackLocal words, local
    __device__ __forceinline__ void push3(WideState& s, int a, bool pa, int b, bool pb, int c, bool pc) {
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
    __device__ __forceinline__ void push_deep(WideState& s, int code) {
        if (s.sp < kStackShared * BLOCK) words[s.sp] = code;
        else if (s.sp < (kStackShared + kStackLocal) * BLOCK) deep[(s.sp - s.base) / BLOCK - kStackShared] = code;
        else {
            s.redo |= kRedoRay;
            return;
        }
        s.sp += BLOCK;
    }
    __device__ __forceinline__ void pop(WideState& s) const {
        if (s.sp == s.base) return;
        s.sp -= BLOCK;
        s.cur = s.sp < kStackShared * BLOCK ? words[s.sp] : deep[(s.sp - s.base) / BLOCK - kStackShared];
    }
};

}  // namespace
}  // namespace wfb
