// Device build of the wide tree (wide_bvh.cuh) from the uploaded preorder nodes. One launch checks the leaves and
// tags their primitives. Then the tree is collapsed level by level, one thread per wide node: a level's nodes are
// numbered after all earlier levels (per-level counts), and each thread hands a child its preorder node in the
// child's own record, so a level needs nothing but the counts of the levels before it. The first levels, up to
// kTopNodes nodes each, run in one block of one launch; each later level is a launch of its own; a small scene's tree
// takes one launch in all. A level costs the latency of its threads' walk over the preorder nodes.
#include <algorithm>
#include <cmath>
#include "engine.hpp"
#include "wide_build.cuh"
#include "../../include/wfb200.h"

namespace wfb {
namespace {

struct WideCtl {
    int bad;                       // some condition of wide_bvh.cuh does not hold
    int top;                       // levels built by wide_build_top
    int count[kWideMaxLevels + 2];  // wide nodes per level
};

// Node i's conditions: box in range and, for a leaf, primitives inside it, each primitive record in one leaf; tags the record
// with the leaf's node id + 1 (the w of its second float4, 0 at upload).
__device__ bool check_leaf(const float4* nodes, int i, float4* prims, int n_spheres) {
    const float4 lo = nodes[2 * i], hi = nodes[2 * i + 1];
    const int leaf = f2i(hi.w);
    bool ok = box_in_range(lo, hi);
    if (leaf >= 0) {
        const int start = leaf >> kLeafCountBits, n = leaf & kLeafCountMask;
        for (int k = 0; k < n; ++k) {
            float4* rec = prims + 3 * (size_t)(start + k);
            ok = ok && prim_in_box(rec, n_spheres, lo, hi);
            ok = (atomicExch(reinterpret_cast<int*>(&rec[1].w), i + 1) == 0) && ok;
        }
        ok = ok && n > 0;
    }
    return ok;
}

// Checks every node; thread 0 starts the tree.
__global__ void wide_check_leaves(const float4* __restrict__ nodes, int nn, float4* prims, int n_spheres,
                                  float4* wide, WideCtl* ctl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        ctl->count[0] = 1;
        reinterpret_cast<int*>(wide)[0] = 0;
    }
    if (i < nn && !check_leaf(nodes, i, prims, n_spheres)) ctl->bad = 1;
}

constexpr int kTopNodes = 128;

// Wide node `at` of a level whose children are numbered from `next` on.
__device__ void build_node(const float4* __restrict__ nodes, int nn, float4* wide, int capacity, int empty, int at,
                           int next, int* next_count, WideCtl* ctl) {
    float4* rec = wide + (size_t)kWideFloat4 * at;
    const int root = *reinterpret_cast<volatile int*>(rec);
    WideKids kids;
    if (!wide_children(nodes, nn, root, &kids)) {
        ctl->bad = 1;
        return;
    }
    int codes[kWideArity], inner = 0;
#pragma unroll
    for (int j = 0; j < kWideArity; ++j) {
        codes[j] = j < kids.n ? f2i(nodes[2 * kids.id[j] + 1].w) : empty;
        inner += codes[j] < 0;
    }
    int id = inner ? next + atomicAdd(next_count, inner) : 0;
#pragma unroll
    for (int j = 0; j < kWideArity; ++j) {
        if (codes[j] >= 0) continue;
        if (id >= capacity) {
            ctl->bad = 1;
            return;
        }
        codes[j] = ~id;
        reinterpret_cast<int*>(wide + (size_t)kWideFloat4 * id)[0] = kids.id[j];
        ++id;
    }
    wide_write(nodes, kids, codes, rec);
}

// One block: levels from the first on while they hold at most `most` nodes.
__device__ void build_levels(const float4* __restrict__ nodes, int nn, float4* wide, int capacity, int empty, int most,
                             WideCtl* ctl) {
    volatile int* count = ctl->count;
    int begin = 0, level = 0;
    for (; level < kWideMaxLevels; ++level) {
        const int n = count[level];
        if (n == 0 || n > most) break;
        for (int i = threadIdx.x; i < n && begin + i < capacity; i += blockDim.x)
            build_node(nodes, nn, wide, capacity, empty, begin + i, begin + n, &ctl->count[level + 1], ctl);
        __threadfence();
        __syncthreads();
        begin += n;
    }
    if (threadIdx.x == 0) ctl->top = level;
}

__global__ void wide_build_top(const float4* __restrict__ nodes, int nn, float4* wide, int capacity, int empty,
                               WideCtl* ctl) {
    build_levels(nodes, nn, wide, capacity, empty, kTopNodes, ctl);
}

// A whole tree of at most kSmallNodes preorder nodes in one block, its nodes in shared memory: leaf check and levels.
constexpr int kSmallNodes = 1024;
__global__ void wide_build_small(const float4* __restrict__ global_nodes, int nn, float4* prims, int n_spheres,
                                 float4* wide, int capacity, int empty, WideCtl* ctl) {
    extern __shared__ float4 nodes[];
    for (int i = threadIdx.x; i < 2 * nn; i += blockDim.x) nodes[i] = global_nodes[i];
    if (threadIdx.x == 0) {
        ctl->count[0] = 1;
        reinterpret_cast<int*>(wide)[0] = 0;
    }
    __threadfence();
    __syncthreads();
    for (int i = threadIdx.x; i < nn; i += blockDim.x)
        if (!check_leaf(nodes, i, prims, n_spheres)) ctl->bad = 1;
    build_levels(nodes, nn, wide, capacity, empty, capacity, ctl);
}

// Level `after_top` of those that wide_build_top left.
__global__ void wide_build_level(const float4* __restrict__ nodes, int nn, float4* wide, int capacity, int empty,
                                 int after_top, WideCtl* ctl) {
    const int level = ctl->top + after_top;
    if (level >= kWideMaxLevels) return;
    int begin = 0;
    for (int l = 0; l < level; ++l) begin += ctl->count[l];
    const int n = ctl->count[level];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n && begin + i < capacity; i += gridDim.x * blockDim.x)
        build_node(nodes, nn, wide, capacity, empty, begin + i, begin + n, &ctl->count[level + 1], ctl);
}

}  // namespace

size_t wide_ctl_bytes() { return (sizeof(WideCtl) + 255) & ~(size_t)255; }

int launch_wide_build(const DevScene& s, float4* prims, int n_prims, float4* wide, int capacity, void* ctl_mem,
                      int first_level, int levels, cudaStream_t stream) {
    WideCtl* ctl = static_cast<WideCtl*>(ctl_mem);
    const int empty = empty_leaf(n_prims);
    (void)cudaGetLastError();  // the check below is for these launches only
    if (first_level == 0) {
        cuda_check(cudaMemsetAsync(ctl, 0, sizeof(WideCtl), stream), "memset wide build");
        if (s.n_nodes <= kSmallNodes) {
            wide_build_small<<<1, 256, (size_t)s.n_nodes * 32, stream>>>(s.nodes, s.n_nodes, prims, s.n_spheres, wide,
                                                                         capacity, empty, ctl);
            cuda_check(cudaGetLastError(), "wide build launch");
            return 0;
        }
        wide_check_leaves<<<(s.n_nodes + 255) / 256, 256, 0, stream>>>(s.nodes, s.n_nodes, prims, s.n_spheres, wide, ctl);
        wide_build_top<<<1, 512, 0, stream>>>(s.nodes, s.n_nodes, wide, capacity, empty, ctl);
        if (levels <= 0) levels = std::max(1, (int)std::ceil(0.62 * std::log2((double)capacity)) - 2);
    }
    if (first_level > 0 && levels <= 0) levels = 8;
    const int grid = std::min((capacity + 63) / 64, 148 * 16);  // 148 SMs, 16 CTAs each: a level strides over the rest
    for (int l = first_level; l < first_level + levels; ++l)
        wide_build_level<<<grid, 64, 0, stream>>>(s.nodes, s.n_nodes, wide, capacity, empty, l, ctl);
    cuda_check(cudaGetLastError(), "wide build launch");
    return first_level + levels;
}

int wide_build_result(const void* ctl_host, int levels_done, bool* finished) {
    const WideCtl* c = static_cast<const WideCtl*>(ctl_host);
    const int done = std::min(c->top + levels_done, kWideMaxLevels);
    *finished = c->bad || c->count[done] == 0 || done == kWideMaxLevels;
    if (c->bad || c->count[done] != 0) return 0;
    long long total = 0;
    for (int l = 0; l < done; ++l) total += c->count[l];
    return (int)total;
}

}  // namespace wfb
