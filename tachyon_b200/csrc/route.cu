// Per-token front end of the MoE block, one CTA per token: (optional) RMSNorm,
// router GEMV, top-k, gating softmax, 8-bit quantization of the row, and - when
// the whole batch fits one CTA's dispatch - the token -> expert dispatch, run by
// whichever CTA finishes last.
//
// Reproduces, value for value:
//   rmsnorm        - src/kernels.rs:522-528 with dot_f32's AVX2 order
//                    (src/kernels_x86.rs:132-154), applied as src/model.rs:662-667;
//   router logits  - Matrix::matmul's bf16 arm (src/weights.rs:230-240) with
//                    the AVX2 dot bf16s (src/kernels_x86.rs:157-171): two
//                    8-lane fma accumulators over 16-element strides, summed
//                    lane-wise, then the fixed hsum tree (33-38);
//   top-k + gates  - route() (src/model.rs:448-457): order by total_cmp
//                    descending, ties to the lower expert, softmax over the k
//                    kept with max = the top score, sum taken in that order;
//   quantization   - quantize_q8 (src/kernels.rs:84-98) per 32-block, as
//                    quantize_input applies it per token (src/weights.rs:652-664).
// The softmax exponential is evaluated in double precision and rounded to
// float; the CPU path calls libm's expf. The two agree except where expf
// itself is not correctly rounded, hence the 1e-5 tolerance on gates.
#include <algorithm>

#include "dispatch_common.cuh"
#include "experts_common.cuh"
#include "route_common.cuh"

namespace tc {

namespace {

constexpr size_t ROUTE_SMEM_LIMIT = 200 * 1024;
constexpr int ROUTE_THREADS = DISPATCH_THREADS;  // the last CTA runs the dispatch with the same threads

struct RouteArgs {
    const uint16_t* router;
    const float* bias;
    const float* x;        // [t, hidden]: the normed input, or the residual stream when norm_w is set
    const float* norm_w;   // RMSNorm weight, or null when x is already normed
    float eps;
    int t, hidden, experts, topk;
    float* logits;
    uint32_t* ids;
    float* gates;
    int8_t* xq;
    float* xs;
    float* xsum;
    // dispatch outputs, used when fused
    int fuse_dispatch;
    int stage_rows;        // tile kernel: rows of the router matrix in shared memory at a time
    int stage_router;      // the router matrix fits in shared memory beside the row: stage it with bulk copies
    int* ticket;
    int* status;
    uint32_t *counts, *offsets, *perm, *pos, *slot_token;
    int* active;
    TokenTile* tiles;      // when set: token tiles of up to tile_cols columns are cut as well
    int *tile_count, tile_cols;
    PeerPlan scatter;      // ranks > 0: the last CTA sends the rows to every rank instead of dispatching
};

__global__ void __launch_bounds__(ROUTE_THREADS) route_kernel(const RouteArgs a) {
    extern __shared__ __align__(128) float smem[];
    float* xrow = smem;                 // [hidden] the block's input row (after the norm)
    float* slog = smem + a.hidden;      // [experts]
    __shared__ float s_inv;
    __shared__ int s_last;
    __shared__ __align__(8) uint64_t s_wbar;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hidden = a.hidden, experts = a.experts, topk = a.topk;
    grid_launch_dependents();
    // The router matrix, one bulk copy per row, into rows padded by 32 bytes (so the four-thread
    // groups of a half-warp read distinct banks). Issued first: it lands while the row is normed.
    const int wstride = 2 * hidden + 32;
    uint8_t* wsm = reinterpret_cast<uint8_t*>(smem) + (size_t(hidden + experts) * 4 + 127) / 128 * 128;
    if (a.stage_router) {
        if (tid == 0) {
            mbar_init(&s_wbar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(&s_wbar, uint32_t(experts) * 2u * uint32_t(hidden));
        }
        __syncthreads();
        if (warp == 0)
            for (int e = lane; e < experts; e += 32)
                bulk_copy(wsm + size_t(e) * wstride, a.router + size_t(e) * hidden, 2 * hidden, &s_wbar);
    }
    // The router matrix is a constant: it streams in while the kernel in front of this
    // one (the previous block's combine) finishes. Everything below reads its output.
    grid_dependency_wait();
    // A CTA walks tokens blockIdx.x, blockIdx.x + gridDim.x, ...: one each for batches of up to a few
    // CTAs per SM, several for prefill-size batches (the staged router matrix is then read once per
    // CTA instead of once per token). The next token's row is requested before this one is worked on.
    bool w_landed = true;
    constexpr int ROW_VEC = 4;  // float4 per thread held ahead: rows of up to 4096 floats
    float4 ahead[ROW_VEC];
    auto request_row = [&](int token) {
#pragma unroll
        for (int i = 0; i < ROW_VEC; i++) {
            const int c = (tid + i * ROUTE_THREADS) * 4;
            if (token < a.t && c < hidden)
                ahead[i] = *reinterpret_cast<const float4*>(a.x + size_t(token) * hidden + c);
        }
    };
    const bool rows_ahead = hidden <= ROW_VEC * ROUTE_THREADS * 4;
    if (rows_ahead) request_row(blockIdx.x);
    for (int token = blockIdx.x; token < a.t; token += gridDim.x) {
        if (token != int(blockIdx.x)) __syncthreads();  // the previous token's row and logits are no longer read
        if (rows_ahead) {
#pragma unroll
            for (int i = 0; i < ROW_VEC; i++) {
                const int c = (tid + i * ROUTE_THREADS) * 4;
                if (c < hidden) *reinterpret_cast<float4*>(xrow + c) = ahead[i];
            }
            request_row(token + gridDim.x);
        } else {
            const float* xin = a.x + size_t(token) * hidden;
            for (int c = tid * 4; c < hidden; c += ROUTE_THREADS * 4)
                *reinterpret_cast<float4*>(xrow + c) = *reinterpret_cast<const float4*>(xin + c);
        }
        __syncthreads();
        if (a.norm_w) route_norm_row(xrow, hidden, a.norm_w, a.eps, &s_inv, tid, ROUTE_THREADS);

        if (a.stage_router && token == int(blockIdx.x)) w_landed = mbar_wait_bounded(&s_wbar, 0);
        route_logits(a.router, a.stage_router && w_landed ? wsm : nullptr, wstride, xrow, a.bias, hidden, 0, experts,
                     slog, a.logits ? a.logits + size_t(token) * experts : nullptr, tid, ROUTE_THREADS);
        __syncthreads();

        // Warp 0 ranks the logits while warps 1.. quantize the row (the two do not depend on each other).
        if (warp == 0)
            route_topk_gates(slog, experts, topk, a.ids + size_t(token) * topk, a.gates + size_t(token) * topk, lane);
        const int padded = (hidden / QK + SUPER - 1) / SUPER * SUPER;
        route_quantize_row(xrow, hidden, a.xq + size_t(token) * hidden, a.xs + size_t(token) * padded,
                           a.xsum + size_t(token) * padded, warp, lane, 1, ROUTE_THREADS / 32 - 1);
    }  // tokens of this CTA

    // ---- the dispatch, by the last CTA to get here (batches of up to one CTA's worth of tokens).
    if (a.stage_router && !w_landed) {
        // The staged copy did not arrive within the spin limit (the logits came from
        // global memory instead). Report it, and give the copy a last bounded chance to
        // land before this shared memory is reused or released.
        if (tid == 0) atomicExch(a.status, ERR_COPY_WAIT_TIMEOUT);
        mbar_wait_bounded(&s_wbar, 0);
    }
    if (a.fuse_dispatch) {
        __threadfence();  // this CTA's ids are visible before its ticket
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(a.ticket, 1) == a.t - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            if (a.scatter.ranks) {
                // Expert parallelism over peer memory: the dispatch runs over every rank's
                // tokens, after this CTA has stored this rank's rows into every window.
                __shared__ uint32_t s_epoch;
                peer_scatter_signal(a.scatter, &s_epoch);
            } else {
                DispatchSmem& sm = *reinterpret_cast<DispatchSmem*>(smem);
                dispatch_small_body(sm, a.ids, a.t, experts, topk, a.counts, a.offsets, a.perm, a.pos,
                                    a.slot_token, a.active, a.status);
                if (a.tiles)
                    token_tiles_body(sm.scount, sm.soff, experts, a.tile_cols, a.tiles, a.tile_count, sm.stiles, sm.srows);
            }
            if (tid == 0) *a.ticket = 0;  // ready for the next launch on this stream
        }
    }
}

// Prefill-size batches: a CTA takes a tile of TILE tokens at a time (walking tiles blockIdx.x,
// blockIdx.x + gridDim.x, ...): a warp per token for the norm, the ranking and the quantization,
// four threads per (TG tokens, ROUTE_TE experts) for the logits, with the router matrix staged once
// per CTA. Same arithmetic per token as route_kernel.
//
// Bound by the shared-memory reads and the latency of a tile's chain (load, norm, logits, ranking). A
// thread's 2 tokens x 2 experts take four reads for four products and keep all eight warps of a CTA busy;
// measured for the whole stage at 4096 tokens of the 1b shape / of 2048 columns and 64 experts: 4 x 1 54 us /
// 154 us, 2 x 2 52 / 148, 4 x 2 52 / 166, 2 x 4 57 / 153 (half the warps idle); 4 x 1 with 512 threads 70 /
// 158. TILE = 8 lets two CTAs share an SM; batches that would then leave SMs without a tile take 4 or 2 (333
// tokens of the 1b shape: 42 tiles of 8, 167 of 2).
constexpr int ROUTE_TE = 2;

// Shared memory of the tile kernel before the staged router matrix: padded rows, logits, norm weight.
__host__ __device__ inline size_t route_tile_bytes(int hidden, int experts, int tile) {
    return (size_t(tile) * (hidden / QK * ROW_PAD_BLOCK + (experts + 3) / 4 * 4) * 4 + size_t(hidden) * 4 + 127) / 128 * 128;
}

template <int TILE>
__global__ void __launch_bounds__(ROUTE_THREADS) route_tile_kernel(const RouteArgs a) {
    constexpr int TG = TILE > 2 ? 2 : 1, TE = ROUTE_TE;
    extern __shared__ __align__(128) float smem[];
    const int hidden = a.hidden, experts = a.experts, topk = a.topk;
    const int rstride = hidden / QK * ROW_PAD_BLOCK;  // floats per padded row
    const int lstride = (experts + 3) / 4 * 4;
    float* xrows = smem;                        // [TILE] padded rows
    float* slog = xrows + TILE * rstride;       // [TILE][lstride]
    float* snw = slog + TILE * lstride;         // [hidden] the norm's weight
    __shared__ __align__(8) uint64_t s_wbar;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_launch_dependents();
    // The router matrix by bulk copies, one per row, into rows padded by 32 bytes: all of it, once, or (a
    // matrix larger than the space left) stage_rows experts at a time, again for every tile.
    const int wstride = 2 * hidden + 32, stage_rows = a.stage_rows;
    uint8_t* wsm = reinterpret_cast<uint8_t*>(smem) + route_tile_bytes(hidden, experts, TILE);
    auto stage = [&](int e_lo) {
        const int n = min(stage_rows, experts - e_lo);
        if (warp == 0) {
            if (lane == 0) mbar_expect_tx(&s_wbar, uint32_t(n) * 2u * uint32_t(hidden));
            __syncwarp();
            for (int e = lane; e < n; e += 32)
                bulk_copy(wsm + size_t(e) * wstride, a.router + size_t(e_lo + e) * hidden, 2 * hidden, &s_wbar);
        }
    };
    if (tid == 0) {
        mbar_init(&s_wbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (a.norm_w)
        for (int c = tid; c < hidden; c += ROUTE_THREADS) snw[c] = a.norm_w[c];  // (a constant: before the wait)
    __syncthreads();
    stage(0);  // (constants as well)
    grid_dependency_wait();
    bool landed = true;
    uint32_t stagings = 0;  // waited for
    const bool once = stage_rows >= experts;
    const int padded = (hidden / QK + SUPER - 1) / SUPER * SUPER;
    const int tiles = (a.t + TILE - 1) / TILE, vec_per_row = hidden / 4;
    const int dk = ROUTE_THREADS / vec_per_row, dv = ROUTE_THREADS - dk * vec_per_row;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int t0 = tile * TILE, nt = min(TILE, a.t - t0);
        __syncthreads();  // the previous tile's rows and logits are no longer read
        const float4* src = reinterpret_cast<const float4*>(a.x + size_t(t0) * hidden);  // (the tile's rows are one run)
        const int vecs = nt * vec_per_row;
        int k = tid / vec_per_row, vc = tid - k * vec_per_row;  // piece i of the run is piece vc of row k
        for (int i0 = 0; i0 < vecs; i0 += ROUTE_THREADS * TILE) {  // all requests of a pass before the first store
            float4 v[TILE];
#pragma unroll
            for (int u = 0; u < TILE; u++) {
                const int i = i0 + u * ROUTE_THREADS + tid;
                if (i < vecs) v[u] = src[i];
            }
#pragma unroll
            for (int u = 0; u < TILE; u++) {
                if (i0 + u * ROUTE_THREADS + tid < vecs)
                    *reinterpret_cast<float4*>(xrows + k * rstride + padded_at(4 * vc)) = v[u];
                k += dk, vc += dv;
                if (vc >= vec_per_row) vc -= vec_per_row, k++;
            }
        }
        __syncthreads();
        if (a.norm_w && warp < nt) {  // a warp per token
            float* xr = xrows + warp * rstride;
            const float ss = __fdiv_rn(sum_squares_padded_row(xr, hidden, lane), float(hidden));
            const float inv = __fdiv_rn(1.0f, __fsqrt_rn(ss + a.eps));
            __syncwarp();
#pragma unroll 8
            for (int c = 0; c < hidden / QK; c++)
                xr[c * ROW_PAD_BLOCK + lane] = xr[c * ROW_PAD_BLOCK + lane] * inv * snw[c * QK + lane];
        }
        for (int e_lo = 0; e_lo < experts; e_lo += stage_rows) {
            if (!once || stagings == 0) {
                landed = mbar_wait_bounded(&s_wbar, stagings & 1) && landed;
                stagings++;
            }
            if (e_lo == 0) __syncthreads();  // the normed rows are complete
            // Logits. Each (token, expert) keeps its own accumulators, as route_dot_quad: thread q of a quad has
            // elements 16 j + 4 q .. + 3. (Rows past the tile's tokens hold anything and experts past the
            // last repeat it; those logits are not stored.)
            const int n_e = min(stage_rows, experts - e_lo), egroups = (n_e + TE - 1) / TE;
            const int tasks = (nt + TG - 1) / TG * egroups;
            for (int p0 = 0; p0 < tasks; p0 += ROUTE_THREADS / 4) {
                const int p = p0 + (tid >> 2), q = tid & 3;
                if (p0 + ((tid >> 5) << 3) >= tasks) continue;  // (a warp without work)
                const bool valid = p < tasks;
                const int grp = valid ? p / egroups : 0, e0 = valid ? (p - grp * egroups) * TE : 0;
                float2 acc[TG][TE][2];
#pragma unroll
                for (int i = 0; i < TG; i++)
#pragma unroll
                    for (int j = 0; j < TE; j++) acc[i][j][0] = acc[i][j][1] = make_float2(0.0f, 0.0f);
                const uint8_t* ws[TE];
#pragma unroll
                for (int j = 0; j < TE; j++) ws[j] = wsm + size_t(min(e0 + j, n_e - 1)) * wstride + q * 8;
                const float* xr = xrows + size_t(grp * TG) * rstride + q * 4;
#pragma unroll 2
                for (int blk = 0; blk < hidden / QK; blk++) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        float4 xv[TG];
#pragma unroll
                        for (int i = 0; i < TG; i++)
                            xv[i] = *reinterpret_cast<const float4*>(xr + i * rstride + blk * ROW_PAD_BLOCK + 16 * h);
#pragma unroll
                        for (int j = 0; j < TE; j++) {
                            const uint2 wv = *reinterpret_cast<const uint2*>(ws[j] + blk * 2 * QK + 32 * h);
                            const float2 w01 = make_float2(bf16_lo(wv.x), bf16_hi(wv.x)), w23 = make_float2(bf16_lo(wv.y), bf16_hi(wv.y));
#pragma unroll
                            for (int i = 0; i < TG; i++) {
                                acc[i][j][0] = fma2(w01, make_float2(xv[i].x, xv[i].y), acc[i][j][0]);
                                acc[i][j][1] = fma2(w23, make_float2(xv[i].z, xv[i].w), acc[i][j][1]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < TG; i++)
#pragma unroll
                    for (int j = 0; j < TE; j++) {
                        // The two 8-lane accumulators added lane-wise, then the hsum tree.
                        const float lanes[4] = {acc[i][j][0].x, acc[i][j][0].y, acc[i][j][1].x, acc[i][j][1].y};
                        float v[4], sv[4];
#pragma unroll
                        for (int l = 0; l < 4; l++) v[l] = lanes[l] + __shfl_xor_sync(0xffffffffu, lanes[l], 2);
#pragma unroll
                        for (int l = 0; l < 4; l++) sv[l] = v[l] + __shfl_xor_sync(0xffffffffu, v[l], 1);
                        float y = (sv[0] + sv[2]) + (sv[1] + sv[3]);
                        y = y + 0.0f;  // the dot's scalar tail is an empty sum
                        const int token = grp * TG + i, e = e_lo + e0 + j;
                        if (valid && q == 0 && token < nt && e0 + j < n_e) {
                            if (a.bias) y = y + a.bias[e];
                            slog[token * lstride + e] = y;
                            if (a.logits) a.logits[size_t(t0 + token) * experts + e] = y;
                        }
                    }
            }
            __syncthreads();
            // The next part of the matrix, for this tile or the next one.
            if (!once && (e_lo + stage_rows < experts || tile + int(gridDim.x) < tiles))
                stage(e_lo + stage_rows < experts ? e_lo + stage_rows : 0);
        }
        if (warp < nt) {  // a warp per token: ranking and gates, then the row's 8-bit blocks
            const size_t token = size_t(t0 + warp);
            route_topk_gates(slog + warp * lstride, experts, topk, a.ids + token * topk, a.gates + token * topk, lane);
            route_quantize_padded_row(xrows + warp * rstride, hidden, a.xq + token * hidden, a.xs + token * padded,
                                      a.xsum + token * padded, lane);
        }
    }
    if (stagings == 0) mbar_wait_bounded(&s_wbar, 0);  // (a CTA without tiles: the copy lands before the memory is released)
    if (!landed) {
        // A copy was late: reported, with a last bounded chance to land.
        mbar_wait_bounded(&s_wbar, (stagings - 1) & 1);
        if (tid == 0) atomicExch(a.status, ERR_COPY_WAIT_TIMEOUT);
    }
}

// One warp per row.
__global__ void rmsnorm_kernel(const float* x, const float* __restrict__ w, float eps, int t, int n,
                               float* out) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= t) return;
    const float* xr = x + size_t(row) * n;
    const float ss = __fdiv_rn(sum_squares_avx_order(xr, n, lane), float(n));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(ss + eps));
    float* o = out + size_t(row) * n;
#pragma unroll 8
    for (int c = lane; c < n; c += 32) o[c] = xr[c] * inv * w[c];
}

}  // namespace

void init_kernels_route() {
    cudaFuncSetAttribute(route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ROUTE_SMEM_LIMIT));
    cudaFuncSetAttribute(route_tile_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ROUTE_SMEM_LIMIT));
    cudaFuncSetAttribute(route_tile_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ROUTE_SMEM_LIMIT));
    cudaFuncSetAttribute(route_tile_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ROUTE_SMEM_LIMIT));
}

int launch_route(const MoeDims& d, const uint16_t* router, const float* bias, const float* x,
                 const float* norm_w, float eps, int t, Workspace& ws, cudaStream_t stream) {
    RouteArgs a{};
    a.router = router;
    a.bias = bias;
    a.x = x;
    a.norm_w = norm_w;
    a.eps = eps;
    a.t = t;
    a.hidden = d.hidden;
    a.experts = d.experts;
    a.topk = d.topk;
    a.logits = ws.logits;
    a.ids = ws.ids;
    a.gates = ws.gates;
    a.xq = ws.xq;
    a.xs = ws.xs;
    a.xsum = ws.xsum;
    a.fuse_dispatch = t <= DISPATCH_THREADS;
    a.ticket = ws.ticket;
    a.status = ws.status;
    a.counts = ws.counts;
    a.offsets = ws.offsets;
    a.perm = ws.perm;
    a.pos = ws.pos;
    a.slot_token = ws.slot_token;
    a.active = ws.active;
    a.tiles = ws.tiles, a.tile_count = ws.tile_count, a.tile_cols = ws.tile_cols;
    if (a.fuse_dispatch) a.scatter = ws.route_scatter;
    size_t smem = (size_t(d.hidden + d.experts) * sizeof(float) + 127) / 128 * 128;
    const size_t staged = smem + size_t(d.experts) * (2 * size_t(d.hidden) + 32);
    a.stage_router = staged <= ROUTE_SMEM_LIMIT;
    if (a.stage_router) smem = staged;
    if (smem < sizeof(DispatchSmem)) smem = sizeof(DispatchSmem);
    const int sms = ws.sms > 0 ? ws.sms : 148;
    if (a.fuse_dispatch) {
        // Up to one CTA's worth of tokens: a CTA per token; the last one to finish runs the dispatch.
        launch_overlapped(route_kernel, dim3(t), dim3(ROUTE_THREADS), smem, stream, a);
    } else {
        // Larger batches: CTAs that walk tiles, as many as stay resident (the staged router matrix is then
        // read a few hundred times, not once per token).
        const size_t wrow = 2 * size_t(d.hidden) + 32;
        int tile = t >= 8 * sms ? 8 : t >= 4 * sms ? 4 : 2;
        while (tile > 2 && route_tile_bytes(d.hidden, d.experts, tile) + 8 * wrow > ROUTE_SMEM_LIMIT) tile /= 2;
        size_t tsmem = route_tile_bytes(d.hidden, d.experts, tile);
        const int fit = int((ROUTE_SMEM_LIMIT - tsmem) / wrow), parts = (d.experts + fit - 1) / fit;
        a.stage_rows = (d.experts + parts - 1) / parts;
        tsmem += size_t(a.stage_rows) * wrow;
        const int per_sm = int(std::max<size_t>(1, std::min<size_t>(4, (220 * 1024) / (tsmem + 1024))));
        const int tiles = (t + tile - 1) / tile;
        launch_overlapped(tile == 8 ? route_tile_kernel<8> : tile == 4 ? route_tile_kernel<4> : route_tile_kernel<2>,
                          dim3(std::min(tiles, per_sm * sms)), dim3(ROUTE_THREADS), tsmem, stream, a);
    }
    int launched = 1;
    // (Expert parallel over peer windows: the dispatch runs later, over every rank's tokens.)
    if (!a.fuse_dispatch && ws.route_scatter.ranks == 0) launched += launch_dispatch(d, t, ws, stream);
    return launched;
}

int launch_rmsnorm(const float* x, const float* w, float eps, int t, int n, float* out,
                   cudaStream_t stream) {
    const int warps = 4;
    rmsnorm_kernel<<<(t + warps - 1) / warps, warps * 32, 0, stream>>>(x, w, eps, t, n, out);
    return 1;
}

}  // namespace tc

