// Token -> expert dispatch: per-expert histogram, prefix scan, and the stable
// permutation of the t*k (token, pick) slots into expert-contiguous order.
//
// The CPU path pushes each token's picks onto per-expert lists while walking
// tokens in order (src/model.rs:474-482), so within an expert the slots are in
// ascending token order and counts[e] is the list length. This file produces
// the same lists without a serial walk. A CTA owns 256 consecutive tokens, a
// thread per token. Each thread sets one bit per pick in a shared bit matrix
// (expert x token); a token's rank among the CTA's earlier tokens that picked
// the same expert is then a popcount of that expert's row below its own bit.
// Per-CTA histograms (row popcounts) are scanned across CTAs for the CTA's
// base, and a warp-shuffle exclusive scan over experts gives each expert's
// first slot.
//
// (Batches above 256 tokens of a layer take the one-kernel form further down; the three passes serve the entry
// point that may be handed ids from anywhere.)
//
// Outputs: counts[E], offsets[E+1], perm[sorted slot] = token*k + j,
// slot_token[sorted slot] = token, pos[token*k + j] = sorted slot, and the
// ascending list of experts that have tokens (active[0..n), active[E] = n),
// which the expert kernels cut into equal shares.
#include <atomic>

#include "dispatch_common.cuh"

namespace tc {

namespace {

// `ids` carries no __restrict__ in the kernels that may wait for other ranks: in the
// peer-memory exchange other GPUs store the ids while the kernel is already resident,
// so the loads must not be treated as reads of memory that never changes.
__global__ void __launch_bounds__(DISPATCH_THREADS)
dispatch_small_kernel(const uint32_t* ids, int t, int experts, int topk,
                      uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets,
                      uint32_t* __restrict__ perm, uint32_t* __restrict__ pos,
                      uint32_t* __restrict__ slot_token, int* __restrict__ active, const PeerWait pw,
                      int* status, TokenTile* tiles, int* tile_count, int tile_cols) {
    __shared__ DispatchSmem sm;
    if (pw.flags) {  // the ids come from other ranks: all of them have signalled this block
        if (int(threadIdx.x) < pw.ranks) peer_wait(pw, threadIdx.x);
        __syncthreads();
    }
    dispatch_small_body(sm, ids, t, experts, topk, counts, offsets, perm, pos, slot_token, active, status);
    if (tiles) token_tiles_body(sm.scount, sm.soff, experts, tile_cols, tiles, tile_count, sm.stiles, sm.srows);
}

// The entry point without allocation, pass 1: each CTA's histogram of its DISPATCH_THREADS tokens.
__global__ void __launch_bounds__(DISPATCH_THREADS)
dispatch_count_kernel(const uint32_t* ids, int t, int experts, int topk,
                      uint32_t* __restrict__ block_hist, int* status) {
    __shared__ uint32_t bits[MAX_EXPERTS][DISPATCH_WARPS];
    const int tid = threadIdx.x;
    mark_picks(bits, ids, blockIdx.x * DISPATCH_THREADS + tid, t, experts, topk, status);
    for (int e = tid; e < experts; e += DISPATCH_THREADS)
        block_hist[size_t(blockIdx.x) * experts + e] = row_count(bits, e);
}

// Pass 2 (one CTA): per expert, scan the CTA histograms into CTA bases; then
// the exclusive scan over experts.
__global__ void __launch_bounds__(DISPATCH_THREADS)
dispatch_scan_kernel(uint32_t* __restrict__ block_hist, int blocks, int experts,
                     uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets,
                     int* __restrict__ active) {
    __shared__ uint32_t scount[MAX_EXPERTS];
    __shared__ uint32_t soff[MAX_EXPERTS + 1];
    const int tid = threadIdx.x;
    for (int e = tid; e < experts; e += DISPATCH_THREADS) {
        uint32_t run = 0;
        for (int b = 0; b < blocks; b++) {
            uint32_t c = block_hist[size_t(b) * experts + e];
            block_hist[size_t(b) * experts + e] = run;
            run += c;
        }
        scount[e] = run;
        counts[e] = run;
    }
    __syncthreads();
    if (tid < 32) scan_experts(scount, soff, experts, tid);
    if (tid >= 32 && tid < 64) list_active(scount, experts, active, tid - 32);
    __syncthreads();
    for (int e = tid; e <= experts; e += DISPATCH_THREADS) offsets[e] = soff[e];
}

// Pass 3: every slot's sorted position. (Bad ids were reported by pass 1.)
__global__ void __launch_bounds__(DISPATCH_THREADS)
dispatch_permute_kernel(const uint32_t* __restrict__ ids, int t, int experts, int topk,
                        const uint32_t* __restrict__ block_base,
                        const uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm,
                        uint32_t* __restrict__ pos, uint32_t* __restrict__ slot_token) {
    __shared__ uint32_t bits[MAX_EXPERTS][DISPATCH_WARPS];
    const int tid = threadIdx.x;
    const int token = blockIdx.x * DISPATCH_THREADS + tid;
    mark_picks(bits, ids, token, t, experts, topk, nullptr);
    if (token < t) {
        for (int q = 0; q < topk; q++) {
            const uint32_t slot = uint32_t(token) * topk + q;
            if (!pick_is_placed(ids, token, q, experts, topk)) continue;
            const int e = ids[slot];
            const uint32_t p = offsets[e] + block_base[size_t(blockIdx.x) * experts + e] +
                               rank_in_cta(bits, e, tid);
            perm[p] = slot;
            slot_token[p] = token;
            pos[slot] = p;
        }
    }
}

}  // namespace

namespace {

// Large batches in one kernel, a CTA per expert: expert e's slots start after all the slots of lower
// experts, so a CTA that counts the ids below e and those equal to e as it reads them needs nothing from the
// others. A warp owns a contiguous range of the slots (read twice: count, then place), which keeps the
// order. The hits of an expert with up to DISPATCH_E_HELD slots go to shared memory first, and the three stores and the
// division by topk are made by a thread per slot. (Made where a hit was found, under a mask in two of three groups of 32
// ids, they were 13 of the kernel's 21 thousand cycles: 4096 tokens of 8 picks of 32 experts 15 us, now 13, of 64 experts
// 16.6, now 14.8.) The slots of an expert with more are placed where they are found: held part by part, they took a walk over
// all ids for every part (router and dispatch of 65536 tokens of 256 columns, 8 picks of 32 experts, 411 us, now 366, with a
// Zipf bias on the router 691, now 399).
// The last CTA to finish lists the experts that have tokens and, when asked, cuts the token tiles.
// (Three passes with a histogram per 256 tokens, most of it launches and a serial scan, against every CTA
// reading all ids, 128 KB from L2: router and dispatch of 4096 tokens of the 1b shape 68 to 58 us.)
constexpr int DISPATCH_E_THREADS = 1024;
constexpr int DISPATCH_E_WARPS = DISPATCH_E_THREADS / 32;
constexpr int DISPATCH_E_HELD = 8192;  // the most slots of an expert that shared memory holds

struct DispatchArgs {
    const uint32_t* ids;
    int slots, experts, topk;
    uint32_t *counts, *offsets, *perm, *pos, *slot_token;
    int* active;
    TokenTile* tiles;
    int* tile_count;
    int tile_cols;
    int *ticket, *status;
};

// The warp's slots of expert e, among lo .. hi - 1, straight to their places: from `at`, before `end`. Not inlined, and the
// other form below a loop that runs once: inlined, or as straight code, the kernel takes 32 registers instead of 51, two CTAs fit an SM,
// both go where the router leaves room first, and router and dispatch of 4096 tokens of the 1b shape take 45 us instead of 40.
__device__ __noinline__ void place_as_found(const uint32_t* ids, uint32_t* perm, uint32_t* slot_token, uint32_t* pos, uint32_t topk,
                                            uint32_t e, int lo, int hi, uint32_t at, uint32_t end) {
    const int lane = threadIdx.x & 31;
    constexpr int HELD = 8;
#pragma unroll 1
    for (int i0 = lo; i0 < hi; i0 += 32 * HELD) {
        uint32_t id[HELD];
#pragma unroll
        for (int u = 0; u < HELD; u++) {
            const int i = i0 + 32 * u + lane;
            id[u] = i < hi ? __ldcg(ids + i) : 0xffffffffu;
        }
#pragma unroll
        for (int u = 0; u < HELD; u++) {
            const uint32_t i = i0 + 32 * u + lane;
            const unsigned ballot = __ballot_sync(0xffffffffu, id[u] == e);
            const uint32_t p = at + __popc(ballot & ((1u << lane) - 1u));
            if (id[u] == e && p < end) perm[p] = i, slot_token[p] = i / topk, pos[i] = p;
            at += __popc(ballot);
        }
    }
}

__global__ void __launch_bounds__(DISPATCH_E_THREADS) dispatch_experts_kernel(const DispatchArgs a, const PeerWait pw) {
    __shared__ uint32_t s_hits[DISPATCH_E_WARPS], s_below[DISPATCH_E_WARPS];
    __shared__ uint32_t s_slots[DISPATCH_E_HELD];
    __shared__ int s_last;
    __shared__ int s_tiles[MAX_EXPERTS / 32], s_rows[MAX_EXPERTS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t e = blockIdx.x;
    grid_launch_dependents();
    grid_dependency_wait();
    if (pw.flags) {  // the ids come from other ranks: all of them have signalled this block
        if (tid < pw.ranks) peer_wait(pw, tid);
        __syncthreads();
    }
    const int per_warp = ((a.slots + DISPATCH_E_WARPS - 1) / DISPATCH_E_WARPS + 31) & ~31;
    const int lo = min(a.slots, warp * per_warp), hi = min(a.slots, lo + per_warp);
    constexpr int HELD = 8;
    auto walk = [&](auto use) {
#pragma unroll 1
        for (int i0 = lo; i0 < hi; i0 += 32 * HELD) {
            uint32_t id[HELD];
#pragma unroll
            for (int u = 0; u < HELD; u++) {
                const int i = i0 + 32 * u + lane;
                id[u] = i < hi ? __ldcg(a.ids + i) : 0xffffffffu;
            }
#pragma unroll
            for (int u = 0; u < HELD; u++) use(i0 + 32 * u + lane, id[u]);
        }
    };
    uint32_t hits = 0, below = 0;
    bool bad = false;
    walk([&](int i, uint32_t id) {
        hits += id == e, below += id < e;
        bad |= i < hi && id >= uint32_t(a.experts);
    });
    hits = __reduce_add_sync(0xffffffffu, hits), below = __reduce_add_sync(0xffffffffu, below);
    if (e == 0 && bad) atomicExch(a.status, ERR_BAD_EXPERT_ID);
    if (lane == 0) s_hits[warp] = hits, s_below[warp] = below;
    __syncthreads();
    const uint32_t h = s_hits[lane], first = __reduce_add_sync(0xffffffffu, s_below[lane]);
    uint32_t at = first + __reduce_add_sync(0xffffffffu, lane < warp ? h : 0u);
    const uint32_t total = __reduce_add_sync(0xffffffffu, h);
    // (The bounds: after a wait for another rank has run out, its ids may still arrive between the two reads.)
    const bool held = total <= uint32_t(DISPATCH_E_HELD);
    if (!held && hits) place_as_found(a.ids, a.perm, a.slot_token, a.pos, a.topk, e, lo, hi, at, first + total);
    for (uint32_t from = first; held && from < first + total; from += DISPATCH_E_HELD) {
        const uint32_t most = min(first + total - from, uint32_t(DISPATCH_E_HELD));
        for (uint32_t k = tid; k < most; k += DISPATCH_E_THREADS) s_slots[k] = 0xffffffffu;  // (none)
        __syncthreads();
        uint32_t p = at - from;
        if (hits) {
            walk([&](int i, uint32_t id) {
                const unsigned ballot = __ballot_sync(0xffffffffu, id == e);
                const uint32_t k = p + __popc(ballot & ((1u << lane) - 1u));
                if (id == e && k < most) s_slots[k] = uint32_t(i);
                p += __popc(ballot);
            });
        }
        __syncthreads();
        for (uint32_t k = tid; k < most; k += DISPATCH_E_THREADS) {
            const uint32_t i = s_slots[k];
            if (i >= uint32_t(a.slots)) continue;
            a.perm[from + k] = i;
            a.slot_token[from + k] = i / uint32_t(a.topk);
            a.pos[i] = from + k;
        }
        __syncthreads();
    }
    if (tid == 0) {
        a.counts[e] = total;
        a.offsets[e] = first;
        if (int(e) == a.experts - 1) a.offsets[a.experts] = first + total;
        __threadfence();
        s_last = atomicAdd(a.ticket, 1) == a.experts - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (tid == 0) *a.ticket = 0;  // ready for the next launch on this stream
    if (a.tiles) token_tiles_body(a.counts, a.offsets, a.experts, a.tile_cols, a.tiles, a.tile_count, s_tiles, s_rows);
    if (warp == DISPATCH_E_WARPS - 1) list_active(a.counts, a.experts, a.active, lane);
}

}  // namespace

int launch_dispatch(const MoeDims& d, int t, Workspace& ws, cudaStream_t stream) {
    if (t <= DISPATCH_THREADS) {
        dispatch_small_kernel<<<1, DISPATCH_THREADS, 0, stream>>>(ws.ids, t, d.experts, d.topk,
                                                                  ws.counts, ws.offsets, ws.perm,
                                                                  ws.pos, ws.slot_token, ws.active,
                                                                  ws.dispatch_wait, ws.status, ws.tiles, ws.tile_count,
                                                                  ws.tile_cols);
        return 1;
    }
    DispatchArgs a{};
    a.ids = ws.ids, a.slots = t * d.topk, a.experts = d.experts, a.topk = d.topk;
    a.counts = ws.counts, a.offsets = ws.offsets, a.perm = ws.perm, a.pos = ws.pos, a.slot_token = ws.slot_token;
    a.active = ws.active;
    a.tiles = ws.tiles, a.tile_count = ws.tile_count, a.tile_cols = ws.tile_cols;
    a.ticket = ws.ticket, a.status = ws.status;
    launch_overlapped(dispatch_experts_kernel, dim3(d.experts), dim3(DISPATCH_E_THREADS), size_t(0), stream, a, ws.dispatch_wait);
    return 1;
}

// ---------------------------------------------------------------------------
// Dispatch for callers that must not allocate.
//
// The three-pass dispatch above needs one piece of scratch besides its inputs
// and outputs: the per-CTA histograms (block_hist). The entry point
// below keeps it in the array that follows, which lives in the
// library's image: every GPU that loads the library holds these 64 KiB until
// the process exits, and no call ever allocates or frees anything.
//
// Limits that follow from the array's size: at most STATIC_MAX_TOKENS tokens
// (64 CTAs of 256) and MAX_EXPERTS experts per call.
//
// The array is shared by every call on a device and keeps whatever the last
// call left in it. Nothing in it has to start at zero: pass 1 overwrites every
// entry that passes 2 and 3 read. Two calls whose kernels overlap on the GPU
// (different streams, or different contexts on one device) would race on it.
//
// What the caller must guarantee about ids: every value below `experts`, and no
// expert named twice by one token. A value that breaks this is not placed (its
// slot is missing from counts, perm and pos) and the next tc_sync reports it.
constexpr int STATIC_MAX_BLOCKS = 64;
constexpr int STATIC_MAX_TOKENS = STATIC_MAX_BLOCKS * DISPATCH_THREADS;
static __device__ __align__(256) uint32_t g_static_block_hist[STATIC_MAX_BLOCKS * MAX_EXPERTS];
// Where the kernels of this entry point report an expert id they refused to place
// (ERR_BAD_EXPERT_ID). Also part of the library's image, for the same reason.
static __device__ int g_static_status;

namespace {
// In host code the arrays' names are only stand-ins; the device addresses come from
// the runtime, once per device. Each slot is written once (to the same value by
// whoever gets there first) and only read afterwards.
constexpr int MAX_DEVICES = 64;
struct StaticAddresses {
    std::atomic<uint32_t*> block_hist{nullptr};
    std::atomic<int*> status{nullptr};
};
StaticAddresses g_static_dev[MAX_DEVICES];
}  // namespace

const char* dispatch_static(int device, const uint32_t* ids, int t, int experts, int topk,
                            uint32_t* counts, uint32_t* offsets, uint32_t* perm, uint32_t* pos,
                            uint32_t* slot_token, int* active, cudaStream_t stream, int** status_word) {
    if (device < 0 || device >= MAX_DEVICES) return "device ordinal out of range";
    if (!ids || !counts || !offsets || !perm || !pos || !slot_token || !active)
        return "an input or output pointer is null";
    if (experts < 1 || experts > MAX_EXPERTS) return "between 1 and 256 experts";
    if (topk < 1 || topk > MAX_TOPK || topk > experts) return "between 1 and min(32, experts) experts per token";
    if (t < 1) return "empty batch";
    if (t > STATIC_MAX_TOKENS) return "more than 16384 tokens: beyond the built-in scratch array";
    // The context's device is made current on every call (and stays current): the launches
    // below and the symbol look-up both act on the current device.
    if (cudaSetDevice(device) != cudaSuccess) return "cudaSetDevice failed";
    StaticAddresses& sa = g_static_dev[device];
    uint32_t* block_hist = sa.block_hist.load(std::memory_order_acquire);
    int* status = sa.status.load(std::memory_order_acquire);
    if (!block_hist || !status) {
        // First call on this device (make it before any stream capture): look the
        // arrays' device addresses up, with this device current.
        void *p = nullptr, *q = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_block_hist) != cudaSuccess || !p)
            return "cudaGetSymbolAddress failed for the built-in scratch array";
        if (cudaGetSymbolAddress(&q, g_static_status) != cudaSuccess || !q)
            return "cudaGetSymbolAddress failed for the built-in status word";
        block_hist = static_cast<uint32_t*>(p);
        status = static_cast<int*>(q);
        sa.block_hist.store(block_hist, std::memory_order_release);
        sa.status.store(status, std::memory_order_release);
    }
    if (status_word) *status_word = status;
    const int blocks = (t + DISPATCH_THREADS - 1) / DISPATCH_THREADS;
    dispatch_count_kernel<<<blocks, DISPATCH_THREADS, 0, stream>>>(ids, t, experts, topk, block_hist, status);
    dispatch_scan_kernel<<<1, DISPATCH_THREADS, 0, stream>>>(block_hist, blocks, experts, counts, offsets, active);
    dispatch_permute_kernel<<<blocks, DISPATCH_THREADS, 0, stream>>>(ids, t, experts, topk, block_hist, offsets,
                                                                     perm, pos, slot_token);
    return cudaGetLastError() == cudaSuccess ? nullptr : "a dispatch kernel failed to launch";
}

}  // namespace tc
