// Persistent megakernel over the ordered traversal (wide_bvh.cuh): the kernel of every scene whose tree has wide nodes.
//
// Work units, jobs, film order, the order of a path's rays and the estimator steps are those of
// megakernel_persistent (megakernel.cu); the films are the same bits, but for the hits that kCullSlack (wide_bvh.cuh)
// leaves open. What differs, and what it is worth (B200,
// icospheres / heightfield 1280x720x16, cornell36 320x180x16; the preorder kernel takes 22.9 / 12.3 / 0.82 ms):
//
//  * Instruction issue bounds it (0.76 of the slots, 15.5 lanes per instruction; DRAM idle): about 790 warp instructions
//    are executed per sample, 40% of them in node steps. So the node step is short (two 32-byte loads,
//    packed multiply-adds, one byte permute per plane, a stack in shared memory): 15.3 -> 14.4 ms against the
//    straightforward form.
//  * The instruction cache came next (1.6 stall cycles per issue; 0.6 now): rays start, paths start and scattering
//    events end at one place each in the code, whatever the lane's material or the reason; cosine and sine are
//    one out-of-line copy. 14.4 / 8.9 / 0.69 -> 13.0 / 8.5 / 0.64 ms. (Path state in a pool of 64 contexts per warp, so
//    that 18 lanes are active per instruction, was slower, 16.2 ms: the pool's bookkeeping and shared memory
//    cost more than the lanes gained.)
//  * 8 CTAs of 128 threads per SM: 64 registers, 17 KB of shared memory (state that only shading reads is parked there,
//    with the stacks). 7 and 6 CTAs spill less but leave the latency of the node chase open (13.0 / 8.7 at 7).
//  * A launch with fewer units than lanes spreads over all warps (64x36x1: 0.162 -> 0.088 ms).
#include <algorithm>
#include "counts.hpp"
#include "engine.hpp"
#include "wide_lane.cuh"
#include "../../include/wfb200.h"

namespace wfb {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBlock = 128;
constexpr int kCtas = 8;

// Words of a path's state that only shading reads, parked in shared memory while its ray is traced (field by field, so
// that a warp's words are consecutive).
enum Field {
    kThr = 0,       // throughput
    kRad = 3,       // radiance so far
    kBits = 6,      // depth | kAliveBit | kSpecularBit
    kPdf = 7,       // prev_pdf
    kKey = 8,
    kDir = 10,      // direction of the next extension ray
    kContrib = 13,  // contribution of the shadow ray under way
    kPixel = 16,
    kSample = 17,
    kJob = 18,      // batch launches only
    kFields = 19
};
constexpr int kDepthMask = (1 << 29) - 1;
constexpr int kAliveBit = 1 << 29;  // the path goes on after its shadow ray
constexpr int kSpecularBit = 1 << 30;

struct WideArgs {
    JobDesc job0;
    const JobDesc* jobs;
    const BatchHeader* hdr;
    DevCounters* counters;
    unsigned int* work;
    int min_active;
    int leaf_batch;
};

template <bool MULTI>
__global__ void __launch_bounds__(kBlock, kCtas) megakernel_wide(const WideArgs a) {
    const int lane = threadIdx.x & 31;
    const unsigned total_units = MULTI ? a.hdr->total_units : a.job0.units;
    const int n_jobs = MULTI ? (int)a.hdr->n_jobs : 1;
    __shared__ float s_park[(MULTI ? kFields : kJob) * kBlock];
    __shared__ int s_stack[kStackShared * kBlock];
    int stack_deep[kStackLocal];
    LaneStack<kBlock> stack{s_stack, stack_deep};
    auto P = [&](int f) -> float& { return s_park[f * kBlock + threadIdx.x]; };

    // ---- the lane's ray ----
    enum { kNoPath = 0, kExtension = 1, kShadow = 2 };
    int kind = kNoPath;
    // A launch with fewer units than lanes spreads them over all warps, the first lanes of each: a warp of few rays ends
    // sooner than one of 32 that diverge.
    const unsigned share = warp_share(total_units, gridDim.x * (kBlock / 32));
    bool out_of_work = (unsigned)lane >= share;
    const int min_active = min(a.min_active, (int)min((share + 1) / 2, 32u));
    wf::Vec3 o{0.f, 0.f, 0.f};
    TravRay ray;
    ray.d = ray.inv_d = wf::Vec3{0.f, 0.f, 0.f};
    WideState ws;
    ws.cur = ws.pend = ws.redo = 0;
    ws.sp = ws.base = threadIdx.x;
    ws.rank = -1;
    ws.best = 0.f;
    const float4 *jwide = nullptr, *jprims = nullptr;
    int jn_spheres = 0;

    for (;;) {
        // ================= traversal: rounds of node steps or of primitive steps =================
        for (;;) {
            const bool in_leaf = ws.pend != 0;
            const bool at_node = ws.cur < 0;
            const unsigned pm = __ballot_sync(kFull, in_leaf);
            const unsigned nm = __ballot_sync(kFull, at_node);
            const int tracing = __popc(pm | nm);
            if (tracing == 0) break;
            if (tracing < min_active) {
                // few lanes left tracing: stop if some other lane has shading or refill to do
                const bool waiting = !(in_leaf || at_node) && (kind != kNoPath || !out_of_work);
                if (__ballot_sync(kFull, waiting) != 0) break;
            }
            const int np = __popc(pm);
            if (np != 0 && (np >= a.leaf_batch || np >= __popc(nm))) {
                if (in_leaf) {
                    wide_prim_step(MULTI ? jprims : a.job0.s.prims, MULTI ? jn_spheres : a.job0.s.n_spheres, o, ray,
                                   kind == kShadow, ws);
                    wide_next(ws, stack);
                }
            } else {
                // two steps per vote, as a loop (unrolled it is slower: more code): 13.03 -> 12.89 ms on icospheres
#pragma unroll 1
                for (int k = 0; k < 2; ++k) {
                    if (ws.cur < 0) {
                        wide_node_step(MULTI ? jwide : a.job0.s.wide, o, ray.inv_d, ws, stack);
                        wide_next(ws, stack);
                    }
                }
            }
        }

        // ================= shading: lanes whose ray has finished; lanes without a path take one =================
        const bool done = ws.cur == 0 && ws.pend == 0;
        bool go_on = false, need = done && kind == kNoPath, fresh = false, shadow_ray = false, alive_after = false;
        int pixel = 0, sample = 0, job = 0;
        wf::PathState ps;
        wf::Vec3 sh_dir{0.f, 0.f, 0.f}, sh_contrib{0.f, 0.f, 0.f};
        float sh_tmax = 0.f;
        if (done && kind != kNoPath) {
            pixel = __float_as_int(P(kPixel));
            sample = __float_as_int(P(kSample));
            if (MULTI) job = __float_as_int(P(kJob));
            const JobDesc& J = MULTI ? a.jobs[job] : a.job0;
            const DevScene& s = J.s;
            const int bits = __float_as_int(P(kBits));
            ps.ray.o = o;
            ps.ray.d = wf::Vec3{P(kDir), P(kDir + 1), P(kDir + 2)};
            ps.ray.tmin = wf::kRayEps;
            ps.ray.tmax = wf::kInf;
            ps.throughput = wf::Vec3{P(kThr), P(kThr + 1), P(kThr + 2)};
            ps.L = wf::Vec3{P(kRad), P(kRad + 1), P(kRad + 2)};
            ps.depth = bits & kDepthMask;
            ps.specular = (bits & kSpecularBit) != 0;
            ps.prev_pdf = P(kPdf);
            ps.key.k0 = __float_as_uint(P(kKey));
            ps.key.k1 = __float_as_uint(P(kKey + 1));
            // the hit preorder traversal returns
            wf::HitRecord h;
            h.t = 0.f;
            h.prim = -1;
            h.u = h.v = 0.f;
            if (!wide_resolve(s.prims, s.nodes, o, ray, kind == kShadow, ws, &h)) {
                const float2 x = exact_trace(s.nodes, s.n_nodes, s.prims, s.n_spheres, o.x, o.y, o.z, ray.d.x, ray.d.y,
                                             ray.d.z, kind == kShadow ? ws.best : wf::kInf, kind == kShadow);
                h.t = x.x;
                h.prim = __float_as_int(x.y);
            }
            bool path_done = false;
            if (kind == kShadow) {
                if (h.prim < 0) ps.L += wf::Vec3{P(kContrib), P(kContrib + 1), P(kContrib + 2)};  // unoccluded
                path_done = (bits & kAliveBit) == 0;
            } else if (!hit_is_valid(s, h)) {
                atomicAdd(&a.counters->invalid_hits, 1u);
                ps.L += ps.throughput * s.env;  // an invalid hit is treated as a miss
                path_done = true;
            } else {
                wf::Surface f;
                wf::Material m;
                const int mat = wf::classify(s, ps, h, J.max_depth, &f, &m);
                path_done = true;
                if (mat >= 0) {
                    wf::Ray sh;
                    int has = 0;
                    const bool alive = wf::shade(s, ps, f, m, mat, &sh, &sh_contrib, &has);
                    path_done = !alive && !has;
                    if (has) {
                        shadow_ray = true;
                        alive_after = alive;
                        sh_dir = sh.d;
                        sh_tmax = sh.tmax;
                    }
                }
            }
            go_on = !path_done;
            if (path_done) {
                // commit the sample; the unit's next one, if there is one, starts in its place
                if (J.chunks > 1) {
                    float* slot = J.lbuf + sample_slot(pixel, sample - J.first_sample, J.film.pixels);
                    slot[0] = ps.L.x;
                    slot[1] = ps.L.y;
                    slot[2] = ps.L.z;
                } else {
                    // one unit holds all samples of the pixel, in order
                    J.film.rgb[3 * pixel] += ps.L.x;
                    J.film.rgb[3 * pixel + 1] += ps.L.y;
                    J.film.rgb[3 * pixel + 2] += ps.L.z;
                    const float l = wf::luminance(ps.L);
                    J.film.lum[pixel] += l;
                    J.film.lum2[pixel] += l * l;
                }
                ++sample;
                const int k = sample - J.first_sample;
                if (J.chunk > 1 && k < J.sample_count && k % J.chunk != 0) fresh = true;
                else need = true;
                kind = kNoPath;
            }
        }
        // units for the lanes that need one: one atomic for the warp
        need = need && !out_of_work;
        const unsigned um = __ballot_sync(kFull, need);
        if (um) {
            const int leader = __ffs(um) - 1;
            unsigned base = 0;
            // batch: the leader finds the job of the warp's first unit and where the next job starts; a lane
            // searches the table itself only when its unit crosses that boundary
            int j0 = 0;
            unsigned next_begin = 0xffffffffu;
            if (lane == leader) {
                base = atomicAdd(a.work, (unsigned)__popc(um));
                if (MULTI && base < total_units) {
                    j0 = job_of_unit(a.jobs, n_jobs, base);
                    if (j0 + 1 < n_jobs) next_begin = a.jobs[j0 + 1].unit_begin;
                }
            }
            base = __shfl_sync(kFull, base, leader);
            if (MULTI) {
                j0 = __shfl_sync(kFull, j0, leader);
                next_begin = __shfl_sync(kFull, next_begin, leader);
            }
            if (need) {
                const unsigned u = base + __popc(um & ((1u << lane) - 1u));
                out_of_work = u >= total_units;
                if (!out_of_work) {
                    if (MULTI) job = u < next_begin ? j0 : job_of_unit(a.jobs, n_jobs, u);
                    const JobDesc& J = MULTI ? a.jobs[job] : a.job0;
                    // unit -> pixel (u mod P) and chunk (u div P): neighbouring lanes, neighbouring pixels
                    const unsigned local = u - J.unit_begin, pixels = (unsigned)J.film.pixels, k = local / pixels;
                    pixel = (int)(local - k * pixels);
                    sample = J.first_sample + (int)k * J.chunk;
                    fresh = true;
                }
            }
        }
        if (fresh) {
            const JobDesc& J = MULTI ? a.jobs[job] : a.job0;
            const int py = pixel / J.s.width;
            ps = wf::init_path(J.s, pixel - py * J.s.width, py, (uint32_t)sample, J.seed);
            shadow_ray = false;
            P(kPixel) = __int_as_float(pixel);
            P(kSample) = __int_as_float(sample);
            P(kKey) = __uint_as_float(ps.key.k0);
            P(kKey + 1) = __uint_as_float(ps.key.k1);
            if (MULTI) {
                P(kJob) = __int_as_float(job);
                jwide = J.s.wide;
                jprims = J.s.prims;
                jn_spheres = J.s.n_spheres;
            }
        }
        if (go_on || fresh) {
            P(kThr) = ps.throughput.x; P(kThr + 1) = ps.throughput.y; P(kThr + 2) = ps.throughput.z;
            P(kRad) = ps.L.x; P(kRad + 1) = ps.L.y; P(kRad + 2) = ps.L.z;
            P(kBits) = __int_as_float(ps.depth | (ps.specular ? kSpecularBit : 0) | (alive_after ? kAliveBit : 0));
            P(kPdf) = ps.prev_pdf;
            P(kDir) = ps.ray.d.x; P(kDir + 1) = ps.ray.d.y; P(kDir + 2) = ps.ray.d.z;
            if (shadow_ray) {
                P(kContrib) = sh_contrib.x; P(kContrib + 1) = sh_contrib.y; P(kContrib + 2) = sh_contrib.z;
            }
            kind = shadow_ray ? kShadow : kExtension;
            o = ps.ray.o;
            wide_begin(shadow_ray ? sh_dir : ps.ray.d, shadow_ray ? sh_tmax : wf::kInf, true, threadIdx.x, &ray, &ws);
        }
        if (__ballot_sync(kFull, kind != kNoPath) == 0) break;
    }
}

template <bool MULTI>
int resident_ctas_wide(int blocks_per_sm) {
    int dev = 0, sms = 0, occ = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, megakernel_wide<MULTI>, kBlock, 0),
               "occupancy");
    if (blocks_per_sm > 0 && blocks_per_sm < occ) occ = blocks_per_sm;
    return sms * std::max(1, occ);
}

}  // namespace

int megakernel_resident_threads(const MegakernelConfig& cfg) { return kBlock * resident_ctas_wide<true>(cfg.blocks_per_sm); }

void launch_megakernel_wide(const JobDesc* job0, const JobDesc* d_jobs, const BatchHeader* d_hdr, DevCounters* counters,
                            unsigned int* work_counter, const MegakernelConfig& cfg, cudaStream_t stream) {
    WideArgs args{};
    if (job0) args.job0 = *job0;
    args.jobs = d_jobs;
    args.hdr = d_hdr;
    args.counters = counters;
    args.work = work_counter;
    args.min_active = cfg.min_active;
    args.leaf_batch = cfg.leaf_batch;
    if (job0) {
        // as many CTAs as are resident; fewer only when there are not as many units as warps
        const long long grid = std::min<long long>(resident_ctas_wide<false>(cfg.blocks_per_sm),
                                                   ((long long)job0->units + kBlock / 32 - 1) / (kBlock / 32));
        megakernel_wide<false><<<(unsigned)std::max<long long>(1, grid), kBlock, 0, stream>>>(args);
    } else {
        megakernel_wide<true><<<(unsigned)resident_ctas_wide<true>(cfg.blocks_per_sm), kBlock, 0, stream>>>(args);
    }
    cuda_check(cudaGetLastError(), "wide megakernel launch");
}

}  // namespace wfb
