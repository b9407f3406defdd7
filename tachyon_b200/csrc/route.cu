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
#include <type_traits>

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
    int stage_router;      // the router matrix fits in shared memory beside the row: stage it with bulk copies
    int part_experts;      // tile kernel: the experts of one CTA (blockIdx.y * part_experts and on)
    int* ticket;
    int* tile_tickets;     // [tiles] the same among the CTAs of a tile
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
    const int token = blockIdx.x;
    const float* xin = a.x + size_t(token) * hidden;
    constexpr int ROW_VEC = 4;  // float4 per thread asked for at a time
    for (int c0 = tid * 4; c0 < hidden; c0 += ROW_VEC * ROUTE_THREADS * 4) {
        float4 v[ROW_VEC];
#pragma unroll
        for (int i = 0; i < ROW_VEC; i++) {
            const int c = c0 + i * ROUTE_THREADS * 4;
            if (c < hidden) v[i] = *reinterpret_cast<const float4*>(xin + c);
        }
#pragma unroll
        for (int i = 0; i < ROW_VEC; i++) {
            const int c = c0 + i * ROUTE_THREADS * 4;
            if (c < hidden) *reinterpret_cast<float4*>(xrow + c) = v[i];
        }
    }
    __syncthreads();
    if (a.norm_w) route_norm_row(xrow, hidden, a.norm_w, a.eps, &s_inv, tid, ROUTE_THREADS);

    const bool w_landed = !a.stage_router || mbar_wait_bounded(&s_wbar, 0);
    route_logits(a.router, a.stage_router && w_landed ? wsm : nullptr, wstride, xrow, a.bias, hidden, 0, experts,
                 slog, a.logits ? a.logits + size_t(token) * experts : nullptr, tid, ROUTE_THREADS);
    __syncthreads();

    // Warp 0 ranks the logits while warps 1.. quantize the row (the two do not depend on each other).
    if (warp == 0)
        route_topk_gates(slog, experts, topk, a.ids + size_t(token) * topk, a.gates + size_t(token) * topk, lane);
    const int padded = (hidden / QK + SUPER - 1) / SUPER * SUPER;
    route_quantize_row(xrow, hidden, a.xq + size_t(token) * hidden, a.xs + size_t(token) * padded,
                       a.xsum + size_t(token) * padded, warp, lane, 1, ROUTE_THREADS / 32 - 1);

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

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Prefill-size batches: a CTA per tile of NG x TG tokens. The logits are a matrix product whose every output is sixteen
// chains of its own (the AVX dot's lanes), so it runs on the FP32 pipe: four threads per TG tokens x TE experts, thread
// q with lanes 4 q .. 4 q + 3, over chunks of KC columns that stand in shared memory twice over. While eight warps work on a
// chunk, eight others bring the next: the rows through registers, normed and quantized on the way, the router's
// by asynchronous copies. Then a warp per token ranks the logits, and every pick gets its gate from a thread of its
// own. More experts than the 64 / NG x TE of a CTA are split over CTAs (SPLIT), whose last one makes the picks.
// (One CTA in several passes over the columns: 256 experts of 1024 columns, router and dispatch, 2500 tokens 278 us, now
// 110, 129 tokens 57, now 25; 128 experts, 4800 tokens 189, now 117; 65 experts, 2500 tokens 91, now 66.)
//
// Bound by shared memory, 16 TG + 8 TE bytes a thread for 2 TG TE packed products: at 4 x 4 a step of sixteen columns is 24
// cycles of it a warp against 16 of the FP32 pipe, at 4 x 8 32 against 32; with whole rows and the whole matrix staged
// (2 x 2, a warp per token for norm, ranking and quantization, one after the other) it was 12 against 4. A step
// takes twice its bound: two warps per scheduler, beside two that bring rows.
// Measured, the kernel alone (us): 4096 tokens of the 1b shape 37 -> 26; 2047 of the 3b shape 42 -> 26; 4096 of 2048 columns
// and 64 experts 138 -> 70; 333 of the 1b shape 12.8 -> 9.7. Where the 26 go, in thousands of cycles: 4 the squares, 30
// the chunks (25 of them products), 6 ranks, 3 gates. Tried: all warps doing both (35), the next step's
// operands requested a step ahead (no change), quantization by four threads a block as the rows come in (twice the instructions).
template <int N>
using Int = std::integral_constant<int, N>;
constexpr int RT_HALF = 256, RT_THREADS = 2 * RT_HALF;  // the threads of either kind

template <int NG, int TG, int TE, int KC>
struct RouteTile {
    static constexpr int TM = NG * TG, EG = RT_HALF / 4 / NG, EP = EG * TE;  // tokens, expert groups, most experts
    static constexpr int XSTRIDE = KC / QK * ROW_PAD_BLOCK;  // floats per staged row piece
    static constexpr int WSTRIDE = KC * 2 + 32;  // bytes per staged router row piece: four neighbouring rows on distinct banks
    static constexpr int X = TM * XSTRIDE * 4, W = EP * WSTRIDE;             // bytes of a buffer
    // Registers: 128 a thread at launch, then split.
    static constexpr int REGS_DOTS = TG * TE > 20 ? 176 : 136, REGS_ROWS = 256 - REGS_DOTS;
    static_assert(KC >= MAX_TOPK, "the exponentials of a tile's picks fit where its rows were");
    __host__ __device__ static int key_stride(int experts) { return (experts + 31) / 32 * 32; }
    static_assert(2 * (X + W) >= int(sizeof(DispatchSmem)), "a dispatch fits where the buffers were");
    __host__ __device__ static size_t bytes(int experts, int topk) {
        return 2 * size_t(X + W) + size_t(TM) * (key_stride(experts) + 2 * topk + 1) * 4;
    }
};

__device__ __forceinline__ float4 four_floats(const float* p) { return make_float4(p[0], p[1], p[2], p[3]); }

template <int NG, int TG, int TE, int KC, bool SPLIT>
__global__ void __launch_bounds__(RT_THREADS, 1) route_tile_kernel(const RouteArgs a) {
    using L = RouteTile<NG, TG, TE, KC>;
    constexpr int TM = L::TM, EG = L::EG, KV = KC / 8;
    constexpr int TASKS = TM * KV, PER = (TASKS + RT_HALF - 1) / RT_HALF;  // eight columns of a row each
    static_assert(TASKS % 32 == 0 && (TASKS <= RT_HALF || RT_HALF % KV == 0), "whole warps, rows evenly");
    extern __shared__ __align__(128) uint8_t rt_smem[];
    const int hidden = a.hidden, experts = a.experts, topk = a.topk, nb = hidden / QK;
    const int kstride = L::key_stride(experts);
    float* xbuf = reinterpret_cast<float*>(rt_smem);              // [2][TM][XSTRIDE]
    uint8_t* wbuf = rt_smem + 2 * L::X;                           // [2][EP][WSTRIDE]
    int* skey = reinterpret_cast<int*>(wbuf + 2 * L::W);          // [TM][kstride] order keys of the logits
    uint32_t* sid = reinterpret_cast<uint32_t*>(skey + TM * kstride);  // [TM][topk] picks
    float* sval = reinterpret_cast<float*>(sid + TM * topk);           // [TM][topk] their scores
    float* sinv = sval + TM * topk;                                    // [TM] 1 / rms
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = blockIdx.x * TM, nt = min(TM, a.t - t0);
    const int padded = (nb + SUPER - 1) / SUPER * SUPER;
    const int chunks = (hidden + KC - 1) / KC;
    const int e_lo = SPLIT ? blockIdx.y * a.part_experts : 0, n_e = SPLIT ? min(a.part_experts, experts - e_lo) : experts;
    const bool first = !SPLIT || blockIdx.y == 0;  // of the tile's CTAs: the one that quantizes
    const bool dots = tid < RT_HALF;
    const int rid = tid - RT_HALF;  // of the threads that bring the rows
    grid_launch_dependents();
    auto stage_router = [&](int c) {
        const int vecs = min(KC, hidden - c * KC) / 8;
        uint8_t* dst = wbuf + (c & 1) * L::W;
#pragma unroll 4
        for (int i = rid; i < n_e * KV; i += RT_HALF) {
            const int e = i / KV, v = i % KV;
            if (v < vecs) cp_async16(dst + e * L::WSTRIDE + v * 16, a.router + size_t(e_lo + e) * hidden + c * KC + v * 8);
        }
        cp_async_commit();
    };
    if (!dots) stage_router(0);  // (a constant: before the wait)
    grid_dependency_wait();

    // ---- 1 / rms of the rows, a warp per token, several at a time
    if (a.norm_w) {
        constexpr int NW = RT_THREADS / 32, AT = TM > NW ? TM / NW : 1;
        if (warp < TM) {
            float acc[AT];
            const float* xr[AT];
#pragma unroll
            for (int i = 0; i < AT; i++) acc[i] = 0.0f, xr[i] = a.x + size_t(t0 + min(warp + NW * i, nt - 1)) * hidden + lane;
#pragma unroll 16
            for (int k = 0; k < nb; k++) {
                float v[AT];
#pragma unroll
                for (int i = 0; i < AT; i++) v[i] = xr[i][k * QK];
#pragma unroll
                for (int i = 0; i < AT; i++) acc[i] = fmaf(v[i], v[i], acc[i]);
            }
#pragma unroll
            for (int i = 0; i < AT; i++) {
                const float ss = __fdiv_rn(fold_squares(acc[i]) + 0.0f, float(hidden));  // (the scalar tail is an empty sum)
                if (lane == 0) sinv[warp + NW * i] = __fdiv_rn(1.0f, __fsqrt_rn(ss + a.eps));
            }
        }
        __syncthreads();
    }

    // ---- logits
    if (!dots) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::REGS_ROWS));
        // This thread stages columns 8 col8 .. of rows row0, row0 + 256 / KV, ... of every chunk.
        const int row0 = rid / KV, col8 = rid % KV;
        const bool stages = rid < TASKS;  // (whole warps)
        // The caller's weight may stand at any float. (Read so from an aligned one too, it is 1 to 2 us of a stage of 20 to 80.)
        const bool norm_vec = reinterpret_cast<uintptr_t>(a.norm_w) % 16 == 0;
        float4 ahead[PER][2], nw[2];
        auto request = [&](int c) {
            const int col = c * KC + col8 * 8;
            const bool on = stages && col < hidden;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                nw[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (on && a.norm_w) nw[h] = norm_vec ? *reinterpret_cast<const float4*>(a.norm_w + col + 4 * h) : four_floats(a.norm_w + col + 4 * h);
#pragma unroll
                for (int i = 0; i < PER; i++) {
                    ahead[i][h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (on)
                        ahead[i][h] = *reinterpret_cast<const float4*>(a.x + size_t(t0 + min(row0 + RT_HALF / KV * i, nt - 1)) * hidden + col + 4 * h);
                }
            }
        };
        auto stage_rows = [&](int c) {
            float* dst = xbuf + (c & 1) * (L::X / 4) + row0 * L::XSTRIDE + col8 / 4 * ROW_PAD_BLOCK + col8 % 4 * 8;
#pragma unroll
            for (int i = 0; i < PER; i++) {
                float4 v[2] = {ahead[i][0], ahead[i][1]};
                if (a.norm_w) {
                    const float inv = sinv[row0 + RT_HALF / KV * i];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        v[h].x = v[h].x * inv * nw[h].x, v[h].y = v[h].y * inv * nw[h].y;
                        v[h].z = v[h].z * inv * nw[h].z, v[h].w = v[h].w * inv * nw[h].w;
                    }
                }
                *reinterpret_cast<float4*>(dst + RT_HALF / KV * i * L::XSTRIDE) = v[0];
                *reinterpret_cast<float4*>(dst + RT_HALF / KV * i * L::XSTRIDE + 4) = v[1];
            }
        };
        // The 8-bit blocks of a chunk that stands in shared memory, a thread per block (with four threads per block, as
        // the rows come in, the divisions cost as many instructions for a quarter of the values), by
        // one half of these warps for the even chunks and the other for the odd ones.
        auto quantize_rows = [&](int c) {
            constexpr int BLOCKS = KC / QK;
            for (int i = rid ^ (c & 1 ? RT_HALF / 2 : 0); i < TM * BLOCKS; i += RT_HALF) {
                const int row = i / BLOCKS, b = c * BLOCKS + i % BLOCKS;
                if (row >= nt || b >= padded) continue;
                const size_t token = size_t(t0 + row);
                float d = 0.0f, su = 0.0f;
                if (b < nb) {
                    const float4* src = reinterpret_cast<const float4*>(xbuf + (c & 1) * (L::X / 4) + row * L::XSTRIDE + i % BLOCKS * ROW_PAD_BLOCK);
                    float4 v[QK / 4];
                    float amax = 0.0f;
#pragma unroll
                    for (int k = 0; k < QK / 4; k++) {
                        v[k] = src[k];
                        amax = fmaxf(fmaxf(fmaxf(fmaxf(amax, fabsf(v[k].x)), fabsf(v[k].y)), fabsf(v[k].z)), fabsf(v[k].w));
                    }
                    d = __fdiv_rn(amax, 127.0f);
                    const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
                    int qsum = 0;
                    uint4* dst = reinterpret_cast<uint4*>(a.xq + token * hidden + size_t(b) * QK);
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        int q0, q1;
                        const uint2 lo = quantize_eight(v[4 * k], v[4 * k + 1], id, q0), hi = quantize_eight(v[4 * k + 2], v[4 * k + 3], id, q1);
                        dst[k] = make_uint4(lo.x, lo.y, hi.x, hi.y);
                        qsum += q0 + q1;
                    }
                    su = d * float(qsum);
                }
                a.xs[token * padded + b] = d, a.xsum[token * padded + b] = su;  // (zeros up to whole super-blocks)
            }
        };
        request(0);
#pragma unroll 1
        for (int c = 0; c <= chunks; c++) {  // chunk c goes in while c - 1 is worked on
            if (c > 0 && c < chunks) stage_router(c);
            if (stages && c < chunks) {
                stage_rows(c);
                if (c + 1 < chunks) request(c + 1);
            }
            if (c > 0 && first) quantize_rows(c - 1);
            cp_async_wait_all();
            __syncthreads();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(L::REGS_DOTS));
        const int quad = tid >> 2, q = tid & 3, tg = quad / EG, eg = quad % EG;  // tokens tg + NG i, experts eg + EG j
        float2 acc[TG][TE][2];
#pragma unroll
        for (int i = 0; i < TG; i++)
#pragma unroll
            for (int j = 0; j < TE; j++) acc[i][j][0] = acc[i][j][1] = make_float2(0.0f, 0.0f);
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < chunks; c++) {
            const float* xr = xbuf + (c & 1) * (L::X / 4) + tg * L::XSTRIDE + q * 4;
            const uint8_t* wr = wbuf + (c & 1) * L::W + eg * L::WSTRIDE + q * 8;
            const int steps = min(KC, hidden - c * KC) / 16;
#pragma unroll(TG * TE < 16 ? 8 : 2)
            for (int s = 0; s < steps; s++) {
                float4 xv[TG];
#pragma unroll
                for (int i = 0; i < TG; i++)
                    xv[i] = *reinterpret_cast<const float4*>(xr + i * NG * L::XSTRIDE + s / 2 * ROW_PAD_BLOCK + s % 2 * 16);
#pragma unroll
                for (int j = 0; j < TE; j++) {  // (experts past the last read what the buffer holds; nothing is made of it)
                    const uint2 w = *reinterpret_cast<const uint2*>(wr + j * EG * L::WSTRIDE + s * 32);
                    const float2 w01 = make_float2(bf16_lo(w.x), bf16_hi(w.x)), w23 = make_float2(bf16_lo(w.y), bf16_hi(w.y));
#pragma unroll
                    for (int i = 0; i < TG; i++) {
                        acc[i][j][0] = fma2(w01, make_float2(xv[i].x, xv[i].y), acc[i][j][0]);
                        acc[i][j][1] = fma2(w23, make_float2(xv[i].z, xv[i].w), acc[i][j][1]);
                    }
                }
            }
            __syncthreads();
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
                const int token = tg + NG * i, e = eg + EG * j;
                if (q == 0 && token < nt && e < n_e) {
                    if (a.bias) y = y + a.bias[e_lo + e];
                    skey[token * kstride + e_lo + e] = total_key(y);
                    if (a.logits) a.logits[size_t(t0 + token) * experts + e_lo + e] = y;
                }
            }
    }
    // Scale rows are padded with zeros to whole super-blocks; those past the last chunk's columns:
    if (!dots && first && padded > chunks * (KC / QK)) {
        const int n = padded - chunks * (KC / QK);
        for (int i = rid; i < nt * n; i += RT_HALF) {
            const size_t at = size_t(t0 + i / n) * padded + chunks * (KC / QK) + i % n;
            a.xs[at] = 0.0f;
            a.xsum[at] = 0.0f;
        }
    }
    __shared__ int s_last;
    auto last_to_get_here = [&](int* ticket, unsigned n) {  // of n CTAs, whose writes the last one then sees
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(ticket, 1) == int(n) - 1;
        __syncthreads();
        if (s_last) __threadfence();
        return s_last != 0;
    };
    // ---- picks and gates
    if (!SPLIT) {
        __syncthreads();  // the keys are complete
        // ranks: larger key first, lower expert first among equals; a warp per token and 32 experts
        const int groups = (experts + 31) / 32;
#pragma unroll 1
        for (int i = warp; i < nt * groups; i += RT_THREADS / 32) {
            const int token = i / groups, g = i - token * groups, e = g * 32 + lane;
            const int* keys = skey + token * kstride;
            const int key = keys[e];
            const int rank = rank_in_order(keys, experts, g, key, e < experts, lane);
            if (e < experts && rank < topk) {
                sid[token * topk + rank] = uint32_t(e);
                sval[token * topk + rank] = __int_as_float(key ^ int(unsigned(key >> 31) >> 1));  // (total_key is its own inverse)
            }
        }
        __syncthreads();
        // gates: softmax over a token's picks, the top score as the maximum, the sum taken in score order
        float* sexp = xbuf;  // (no longer read)
        for (int i = tid; i < nt * topk; i += RT_THREADS) sexp[i] = exp_nonpositive_f64(sval[i] - sval[i / topk * topk]);
        __syncthreads();
        for (int i = tid; i < nt * topk; i += RT_THREADS) {
            const float* ex = sexp + i / topk * topk;
            float sum = 0.0f;
            for (int j = 0; j < topk; j++) sum = sum + ex[j];
            a.ids[size_t(t0) * topk + i] = sid[i];
            a.gates[size_t(t0) * topk + i] = __fdiv_rn(sexp[i], sum);
        }
    } else {
        // By the last of the tile's CTAs, from the logits as they all stored them, a warp per token. (The ranking above grows with
        // the square of the experts: every key against every other.)
        if (!last_to_get_here(a.tile_tickets + blockIdx.x, gridDim.y)) return;
        if (tid == 0) a.tile_tickets[blockIdx.x] = 0;  // ready for the next launch on this stream
        float* slog = reinterpret_cast<float*>(skey);
        for (int token = warp; token < nt; token += RT_THREADS / 32) {
            for (int e = lane; e < experts; e += 32) slog[token * kstride + e] = __ldcg(a.logits + size_t(t0 + token) * experts + e);
            __syncwarp();
            const size_t at = size_t(t0 + token) * topk;
            route_topk_gates(slog + token * kstride, experts, topk, a.ids + at, a.gates + at, lane);
        }
    }
    // ---- the dispatch of a batch that one CTA can dispatch, by the last CTA to get here (its first 256 threads have a token
    // each; the others take part in the barriers)
    if (a.fuse_dispatch && last_to_get_here(a.ticket, gridDim.x)) {
        DispatchSmem& sm = *reinterpret_cast<DispatchSmem*>(rt_smem);
        dispatch_small_body(sm, a.ids, a.t, experts, topk, a.counts, a.offsets, a.perm, a.pos, a.slot_token, a.active, a.status);
        if (a.tiles) token_tiles_body(sm.scount, sm.soff, experts, a.tile_cols, a.tiles, a.tile_count, sm.stiles, sm.srows);
        if (tid == 0) *a.ticket = 0;  // ready for the next launch on this stream
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
    auto opt_in = [](auto kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ROUTE_SMEM_LIMIT)); };
    auto every_width = [&](auto split) {
        constexpr bool S = decltype(split)::value;
        opt_in(route_tile_kernel<8, 4, 5, 128, S>), opt_in(route_tile_kernel<8, 4, 8, 128, S>);
        opt_in(route_tile_kernel<8, 2, 5, 128, S>), opt_in(route_tile_kernel<8, 2, 8, 128, S>);
        opt_in(route_tile_kernel<8, 1, 5, 256, S>), opt_in(route_tile_kernel<8, 1, 8, 256, S>);
        opt_in(route_tile_kernel<4, 1, 3, 512, S>), opt_in(route_tile_kernel<4, 1, 4, 512, S>);
    };
    every_width(std::false_type{}), every_width(std::true_type{});
    opt_in(route_tile_kernel<8, 4, 4, 128, false>), opt_in(route_tile_kernel<8, 2, 4, 128, false>);
    opt_in(route_tile_kernel<8, 1, 4, 256, false>), opt_in(route_tile_kernel<4, 1, 2, 512, false>);
}

// The most tiles of a launch: as many as run at once, or tiles of 32.
size_t route_tile_tickets(int max_tokens, int sms) { return size_t(std::max(sms, max_tokens / 32 + 1)); }

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
    a.tile_tickets = ws.tile_tickets;
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
    if (a.fuse_dispatch && (t <= 128 || a.scatter.ranks > 0)) {
        // Few tokens (or rows that go to every rank from here): a CTA per token; the last one to finish runs the dispatch.
        // (Past 128 the tiles below are ahead, whole blocks of 129 / 200 / 256 tokens in us: 1b shape 69.9 / 74.9 / 87.6 so,
        // 67.5 / 71.0 / 82.8 in tiles; 64 experts of 2048 x 1024 201 / 205 / 211, 196 / 200 / 205. Up to 128 these kernels run
        // where the one-kernel block does not: switched off, the CPU's order of lanes, the two matrices in different formats, rows
        // longer than it takes.)
        launch_overlapped(route_kernel, dim3(t), dim3(ROUTE_THREADS), smem, stream, a);
    } else {
        // A CTA per tile of 4, 8, 16 or 32 tokens and up to 64 experts: the narrowest tile whose CTAs all run at once (one
        // fills an SM), else the widest, whose products cost the fewest bytes of shared memory. The line lies where a second
        // wave begins: router and dispatch of the 1b shape in us, one wave of the wider tile / two of the narrower, at 600 tokens 23 / 25,
        // 1300 29 / 32, 2500 38 / 43; 64 experts of 2048 columns 37 / 43, 53 / 62, 79 / 93.
        const int parts = (d.experts + 63) / 64;
        a.part_experts = (d.experts + parts - 1) / parts;
        int tm = 4;
        while (tm < 32 && (t + tm - 1) / tm * parts > sms) tm *= 2;
        auto tile = [&](auto ng, auto tg, auto te, auto kc, auto split) {
            constexpr int NG = decltype(ng)::value, TG = decltype(tg)::value, TE = decltype(te)::value, KC = decltype(kc)::value;
            launch_overlapped(route_tile_kernel<NG, TG, TE, KC, decltype(split)::value>, dim3((t + tm - 1) / tm, parts),
                              dim3(RT_THREADS), RouteTile<NG, TG, TE, KC>::bytes(d.experts, d.topk), stream, a);
        };
        // (Experts cut in parts are 33 to 64 each. Between the widths for 32 and for 64 lies one that fits 40, or 48 where sixteen threads
        // share the experts: with the widest instead, router and dispatch of 40 experts of 1536 columns take 31 us, so 27, at 600 tokens, 66
        // and 58 at 4096; of 48 experts of 1024 columns 22.9 and 21.2 at 129 tokens.)
        auto widths = [&](auto split) {
            const int n = a.part_experts;
            if (tm == 4) n <= 48 ? tile(Int<4>{}, Int<1>{}, Int<3>{}, Int<512>{}, split) : tile(Int<4>{}, Int<1>{}, Int<4>{}, Int<512>{}, split);
            else if (tm == 8) n <= 40 ? tile(Int<8>{}, Int<1>{}, Int<5>{}, Int<256>{}, split) : tile(Int<8>{}, Int<1>{}, Int<8>{}, Int<256>{}, split);
            else if (tm == 16) n <= 40 ? tile(Int<8>{}, Int<2>{}, Int<5>{}, Int<128>{}, split) : tile(Int<8>{}, Int<2>{}, Int<8>{}, Int<128>{}, split);
            else n <= 40 ? tile(Int<8>{}, Int<4>{}, Int<5>{}, Int<128>{}, split) : tile(Int<8>{}, Int<4>{}, Int<8>{}, Int<128>{}, split);
        };
        const std::false_type whole;
        if (parts > 1) widths(std::true_type{});
        else if (d.experts > 32) widths(whole);
        else if (tm == 4) tile(Int<4>{}, Int<1>{}, Int<2>{}, Int<512>{}, whole);
        else if (tm == 8) tile(Int<8>{}, Int<1>{}, Int<4>{}, Int<256>{}, whole);
        else if (tm == 16) tile(Int<8>{}, Int<2>{}, Int<4>{}, Int<128>{}, whole);
        else tile(Int<8>{}, Int<4>{}, Int<4>{}, Int<128>{}, whole);
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

