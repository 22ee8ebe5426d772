// Stand-alone queue primitives behind the C ABI (include/wfb200.h), replacing the reference's
// scan_workspace_create / scan_exclusive_u32 / compact_u32 / test_queue_push
// (WVM/src/gpu/queues.cuh:30-55, WVM/src/gpu/queues.cu:99-252) with single-pass kernels:
//   scan     one launch, one read and one write per element (decoupled look-back), in-place safe;
//   compact  one launch: flags -> tile scan -> stable scatter (no indicator array, no second pass).
// Tiles are claimed through an atomic ticket, so a tile only ever waits on tiles claimed before
// it by CTAs that are already running: the look-back always makes progress.
#include <atomic>
#include <cstring>
#include "counts.hpp"
#include "engine.hpp"
#include "queues.cuh"
#include "queues.hpp"
#include "../../include/wfb200.h"

namespace wfb {
namespace {

constexpr int kScanBlock = 256;
constexpr int kScanWarps = kScanBlock / 32;
// A warp's part of a tile is a run of chunks of 128 elements: lane l holds elements 4 l .. 4 l + 3 of each, one 16-byte
// access per chunk (4-byte ones for arrays that do not start on 16 bytes, and at the end). Chunks per warp: 4 for
// arrays that then still fill the SMs with tiles, 1 for shorter ones.
//
// Both kernels are bound by memory: 16,000,003 flags and values, 40% kept, on a B200 with the L2 flushed, take 34.7 us for
// the scan (128 MB, 3.7 TB/s) and 45.1 us for the compaction (154 MB, 3.4 TB/s; the kept values leave through shared
// memory, in order), where tiles of 1024 with one element per access took 73.8 and 83.9; 1,000 elements 6.1 us
// (8.0 with a launch to reset the tickets). 2 and 8 chunks per warp: 43.0 / 47.2 and 32.7 / 46.0 us.
constexpr int kChunk = 128;
constexpr int kLargeChunks = 4;
constexpr int kLargeScan = 1 << 20;  // elements; at 4096 a tile, 256 CTAs and more
template <int CHUNKS>
constexpr int kTileElements = kScanWarps * kChunk * CHUNKS;
constexpr int kSmallTile = kTileElements<1>;

// The 4 elements at i (i a multiple of 4) of an array of n, 0 past its end.
__device__ __forceinline__ uint4 load4(const uint32_t* p, long long i, int n, bool aligned) {
    if (aligned && i + 4 <= n) return *reinterpret_cast<const uint4*>(p + i);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (i < n) v.x = p[i];
    if (i + 1 < n) v.y = p[i + 1];
    if (i + 2 < n) v.z = p[i + 2];
    if (i + 3 < n) v.w = p[i + 3];
    return v;
}

// MODE 0: exclusive scan of in[] into out[] (in may equal out), *total = sum.
// MODE 1: stable compaction: out[k] = values[i] for the k-th i with flags[i] != 0, *total = count.
// `aligned`: in, values and (MODE 0) out start on 16 bytes. Tickets run from first_ticket on; the CTA that takes the last
// one puts the counter back, so no launch has to reset it.
template <int MODE, int CHUNKS>
__global__ void __launch_bounds__(kScanBlock) scan_tiles(const uint32_t* in, const uint32_t* values, uint32_t* out,
                                                         int n, uint32_t* total, unsigned long long* status,
                                                         unsigned* ticket, unsigned first_ticket, bool aligned,
                                                         unsigned epoch, unsigned* err, unsigned long long wait_ns) {
    constexpr int kTile = kTileElements<CHUNKS>;
    __shared__ uint32_t s_warp[kScanWarps];
    __shared__ int s_tile;
    __shared__ uint32_t s_prefix;
    __shared__ uint32_t s_kept[MODE == 1 ? kTile : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(ticket, 1u);
        if (t == first_ticket + gridDim.x - 1) atomicExch(ticket, 0u);
        s_tile = (int)t;
    }
    __syncthreads();
    const int tile = s_tile;
    const long long base = (long long)tile * kTile + (long long)warp * (kChunk * CHUNKS) + lane * 4;
    uint4 x[CHUNKS], val[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) x[c] = load4(in, base + c * kChunk, n, aligned);  // before any write: in-place safe
    if (MODE == 1) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) val[c] = load4(values, base + c * kChunk, n, aligned);
    }
    // exclusive prefix of each of the lane's 4-element groups within the warp's part
    uint32_t before[CHUNKS];
    uint32_t warp_sum = 0;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        if (MODE == 1) x[c] = make_uint4(x[c].x != 0u, x[c].y != 0u, x[c].z != 0u, x[c].w != 0u);
        const uint32_t s = x[c].x + x[c].y + x[c].z + x[c].w;
        const uint32_t inc = warp_inclusive_sum(s);
        before[c] = warp_sum + inc - s;
        warp_sum += __shfl_sync(kFullMask, inc, 31);
    }
    if (lane == 0) s_warp[warp] = warp_sum;
    __syncthreads();
    uint32_t warp_before = 0, aggregate = 0;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) {
        const uint32_t t = s_warp[w];
        warp_before += w < warp ? t : 0u;
        aggregate += t;
    }
    if (threadIdx.x == 0) publish_status(status, tile, epoch, tile == 0 ? kStatusPrefix : kStatusAggregate, aggregate);
    if (MODE == 1) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            uint32_t at = warp_before + before[c];
            if (x[c].x) s_kept[at++] = val[c].x;
            if (x[c].y) s_kept[at++] = val[c].y;
            if (x[c].z) s_kept[at++] = val[c].z;
            if (x[c].w) s_kept[at++] = val[c].w;
        }
    }
    if (tile > 0 && warp == 0) {
        const uint32_t p = tile_lookback(status, tile, epoch, err, wait_ns);
        if (lane == 0) {
            publish_status(status, tile, epoch, kStatusPrefix, p + aggregate);
            s_prefix = p;
        }
    } else if (tile == 0 && threadIdx.x == 0) {
        s_prefix = 0;
    }
    __syncthreads();
    const uint32_t prefix = s_prefix;
    if (MODE == 1) {
        for (uint32_t k = threadIdx.x; k < aggregate; k += kScanBlock) out[prefix + k] = s_kept[k];
    } else {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const long long i = base + c * kChunk;
            uint4 y;
            y.x = prefix + warp_before + before[c];
            y.y = y.x + x[c].x;
            y.z = y.y + x[c].y;
            y.w = y.z + x[c].z;
            if (aligned && i + 4 <= n) {
                *reinterpret_cast<uint4*>(out + i) = y;
            } else {
                if (i < n) out[i] = y.x;
                if (i + 1 < n) out[i + 1] = y.y;
                if (i + 2 < n) out[i + 2] = y.z;
                if (i + 3 < n) out[i + 3] = y.w;
            }
        }
    }
    if (total && (long long)(tile + 1) * kTile >= n && threadIdx.x == 0) *total = prefix + aggregate;
}

__global__ void queue_push_test_kernel(const uint32_t* flags, int n, uint32_t* items, uint32_t capacity,
                                       uint32_t* counter, uint32_t* overflow) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool pred = i < n && flags[i] != 0u;
    queue_push(items, counter, capacity, (uint32_t)i, pred, overflow);
}

std::atomic<unsigned long long> g_wait_limit_ns{kDefaultWaitLimitNs};
std::atomic<bool> g_unsatisfiable_next{false};

// Tile tickets start at 0; a test that asked for an unsatisfiable wait starts them at 1, so no CTA
// claims tile 0 and every look-back waits for a prefix that nothing publishes.
unsigned start_tickets(ScanWorkspace& ws, cudaStream_t stream) {
    if (!take_unsatisfiable_wait()) return 0u;
    static const unsigned one = 1u;
    cuda_check(cudaMemcpyAsync(ws.ticket, &one, sizeof(unsigned), cudaMemcpyHostToDevice, stream), "set ticket");
    cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");  // `one` is read before returning
    return 1u;
}

template <int MODE>
void launch_scan(const uint32_t* in, const uint32_t* values, uint32_t* out, int n, uint32_t* total, ScanWorkspace& ws,
                 cudaStream_t stream) {
    const unsigned first = start_tickets(ws, stream);
    const unsigned epoch = ++ws.epoch;
    uintptr_t bits = reinterpret_cast<uintptr_t>(in);
    bits |= MODE == 1 ? reinterpret_cast<uintptr_t>(values) : reinterpret_cast<uintptr_t>(out);
    const bool aligned = (bits & 15) == 0;
    const bool large = n >= kLargeScan;
    const int tile = large ? kTileElements<kLargeChunks> : kSmallTile;
    const int tiles = scan_tile_count(n, tile);
    const auto kernel = large ? scan_tiles<MODE, kLargeChunks> : scan_tiles<MODE, 1>;
    (void)cudaGetLastError();  // the check below is for this launch only
    kernel<<<tiles, kScanBlock, 0, stream>>>(in, values, out, n, total, ws.status, ws.ticket, first, aligned, epoch,
                                             ws.err, device_wait_limit_ns());
    cuda_check(cudaGetLastError(), MODE == 0 ? "scan launch" : "compact launch");
}

}  // namespace

uint64_t device_wait_limit_ns() { return g_wait_limit_ns.load(); }

void set_device_wait_test(uint64_t limit_ns, bool unsatisfiable_next) {
    g_wait_limit_ns.store(limit_ns ? limit_ns : kDefaultWaitLimitNs);
    g_unsatisfiable_next.store(unsatisfiable_next);
}

bool take_unsatisfiable_wait() { return g_unsatisfiable_next.exchange(false); }

ScanWorkspace::~ScanWorkspace() {
    if (arena) cudaFree(arena);
}

std::unique_ptr<ScanWorkspace> scan_workspace_create(int capacity) {
    if (capacity <= 0) throw Error(WFB_ERR_INVALID_ARGUMENT, "scan workspace capacity must be positive");
    auto ws = std::make_unique<ScanWorkspace>();
    const size_t tiles = ((size_t)capacity + kSmallTile - 1) / kSmallTile + 2;
    const size_t bytes = 256 + tiles * sizeof(unsigned long long);
    cuda_check(cudaMalloc(&ws->arena, bytes), "cudaMalloc scan workspace");
    cuda_check(cudaMemset(ws->arena, 0, bytes), "cudaMemset scan workspace");
    ws->ticket = static_cast<unsigned*>(ws->arena);
    ws->err = ws->ticket + 1;
    ws->status = reinterpret_cast<unsigned long long*>(static_cast<char*>(ws->arena) + 256);
    ws->capacity = capacity;
    ws->bytes = bytes;
    return ws;
}

void scan_exclusive_u32(const uint32_t* in, uint32_t* out, int n, uint32_t* total, ScanWorkspace& ws,
                        cudaStream_t stream) {
    if (n < 0 || n > ws.capacity) throw Error(WFB_ERR_INVALID_ARGUMENT, "scan size exceeds the workspace capacity");
    if (n == 0) {
        if (total) cuda_check(cudaMemsetAsync(total, 0, sizeof(uint32_t), stream), "memset total");
        return;
    }
    launch_scan<0>(in, nullptr, out, n, total, ws, stream);
}

void compact_u32(const uint32_t* values, const uint32_t* flags, uint32_t* out, uint32_t* count, int n,
                 ScanWorkspace& ws, cudaStream_t stream) {
    if (n < 0 || n > ws.capacity) throw Error(WFB_ERR_INVALID_ARGUMENT, "compaction size exceeds the workspace capacity");
    if (n == 0) {
        if (count) cuda_check(cudaMemsetAsync(count, 0, sizeof(uint32_t), stream), "memset count");
        return;
    }
    launch_scan<1>(flags, values, out, n, count, ws, stream);
}

void test_queue_push(const uint32_t* flags, int n, uint32_t* items, uint32_t capacity, uint32_t* counter,
                     uint32_t* overflow, cudaStream_t stream) {
    if (n < 0) throw Error(WFB_ERR_INVALID_ARGUMENT, "negative size");
    if (n == 0) return;
    queue_push_test_kernel<<<(n + 255) / 256, 256, 0, stream>>>(flags, n, items, capacity, counter, overflow);
    cuda_check(cudaGetLastError(), "queue push launch");
}

bool scan_workspace_failed(ScanWorkspace& ws, cudaStream_t stream) {
    unsigned e = 0;
    cuda_check(cudaMemcpyAsync(&e, ws.err, sizeof(e), cudaMemcpyDeviceToHost, stream), "read scan error flag");
    cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
    return e != 0;
}

}  // namespace wfb
