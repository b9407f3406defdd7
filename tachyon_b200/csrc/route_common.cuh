// The per-token front end of the MoE block as device functions, shared by the
// stand-alone router kernel (route.cu) and the one-kernel decode block
// (moe_decode.cu): RMSNorm, router logits, top-k with gating softmax, and the
// 8-bit quantization of the token's row.
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
// The softmax exponential is evaluated in double precision (a short polynomial of
// this file, accurate to about 1e-16) and rounded to float; the CPU path calls libm's
// expf. The two agree except where expf itself is not correctly rounded, hence the
// 1e-5 tolerance on gates.
#pragma once

#include "common.cuh"

namespace tc {

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// f32::total_cmp as an integer key (larger key = later in total order).
__device__ __forceinline__ int total_key(float v) {
    int b = __float_as_int(v);
    return b ^ int(unsigned(b >> 31) >> 1);
}

// The hsum tree of src/kernels_x86.rs:33-38 over 8 values held by lanes
// j..j+7 of an aligned 8-lane group: (v0+v4, v1+v5, v2+v6, v3+v7) ->
// (s0+s2, s1+s3) -> s0+s1. Lane j%8==0 ends with the sum.
__device__ __forceinline__ float hsum8(float v, unsigned mask) {
    v = v + __shfl_down_sync(mask, v, 4, 8);
    v = v + __shfl_down_sync(mask, v, 2, 8);
    v = v + __shfl_down_sync(mask, v, 1, 8);
    return v;
}

// The end of the sum of squares below: the four 8-lane accumulators that the lanes hold side by side, (acc0+acc1)+(acc2+acc3)
// lane-wise, then the hsum tree. Lane 0 ends with the sum.
__device__ __forceinline__ float fold_squares(float acc) {
    float s = acc + __shfl_down_sync(0xffffffffu, acc, 8);  // lanes 0-7: a0+a1; 16-23: a2+a3
    s = s + __shfl_down_sync(0xffffffffu, s, 16);           // lanes 0-7: the four summed
    return hsum8(s, 0xffffffffu);
}

// Sum of squares of a row in dot_f32's order, by one warp: lane L owns the
// elements L, L+32, ... (the four 8-lane accumulators of the main loop side by
// side); leftover groups of eight go to the first accumulator; then
// (acc0+acc1)+(acc2+acc3) lane-wise, the hsum tree, and the scalar tail.
__device__ __forceinline__ float sum_squares_avx_order(const float* xr, int n, int lane) {
    float acc = 0.0f;
    int i = 0;
#pragma unroll 16
    for (; i + 32 <= n; i += 32) {
        const float v = xr[i + lane];
        acc = fmaf(v, v, acc);
    }
    for (; i + 8 <= n; i += 8) {
        if (lane < 8) {
            const float v = xr[i + lane];
            acc = fmaf(v, v, acc);
        }
    }
    float s = fold_squares(acc);
    float tail = 0.0f;
    for (int j = i; j < n; j++) tail = tail + xr[j] * xr[j];
    s = s + tail;
    return __shfl_sync(0xffffffffu, s, 0);
}

// xrow[0..hidden) (shared memory, already loaded) becomes rmsnorm(xrow) * norm_w. Called
// by every thread of the CTA; s_inv is one shared float. Ends with a CTA barrier.
__device__ __forceinline__ void route_norm_row(float* xrow, int hidden, const float* norm_w, float eps,
                                               float* s_inv, int tid, int nthreads) {
    if ((tid >> 5) == 0) {
        const float ss = __fdiv_rn(sum_squares_avx_order(xrow, hidden, tid & 31), float(hidden));
        if (tid == 0) *s_inv = __fdiv_rn(1.0f, __fsqrt_rn(ss + eps));
    }
    __syncthreads();
    const float inv = *s_inv;
    for (int c = tid; c < hidden; c += nthreads) xrow[c] = xrow[c] * inv * norm_w[c];
    __syncthreads();
}

// One router logit: dot(bf16 row of expert e, xrow) by FOUR threads (q = 0..3 of an aligned
// quad), each holding four of the dot's sixteen float lanes: thread q owns elements
// 16j+4q..16j+4q+3, so q = 0,1 hold the first 8-lane accumulator of the AVX2 dot and q = 2,3
// the second. `staged`: the router matrix in shared memory with rows `wstride` bytes apart (row
// index e_staged), or null to read expert e's row from global memory (a whole batch of steps
// is requested before the chains run, so the loads overlap instead of each waiting for the
// previous fma). A warp none of whose quads has work passes busy = false and skips the loop (it
// would only take shared-memory bandwidth from the warps that have work) but still takes part
// in the shuffles. The value is complete in every thread of the quad.
__device__ __forceinline__ float route_dot_quad(const uint16_t* router, const uint8_t* staged, int wstride,
                                                const float* xrow, int hidden, int e, int q, bool busy,
                                                int e_staged = -1) {
    constexpr int BATCH = 8;
    const uint16_t* w = router + size_t(e) * hidden + q * 4;
    const float* xr = xrow + q * 4;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (!busy) {
    } else if (staged) {
        const uint8_t* ws = staged + size_t(e_staged >= 0 ? e_staged : e) * wstride + q * 8;
#pragma unroll 16
        for (int c = 0; c < hidden; c += 16) {
            const uint2 wv = *reinterpret_cast<const uint2*>(ws + 2 * c);
            const float4 xv = *reinterpret_cast<const float4*>(xr + c);
            acc[0] = fmaf(bf16_lo(wv.x), xv.x, acc[0]);
            acc[1] = fmaf(bf16_hi(wv.x), xv.y, acc[1]);
            acc[2] = fmaf(bf16_lo(wv.y), xv.z, acc[2]);
            acc[3] = fmaf(bf16_hi(wv.y), xv.w, acc[3]);
        }
    } else {
        for (int c0 = 0; c0 < hidden; c0 += 16 * BATCH) {
            uint2 wv[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; u++)
                wv[u] = c0 + 16 * u < hidden ? __ldg(reinterpret_cast<const uint2*>(w + c0 + 16 * u))
                                             : make_uint2(0u, 0u);
#pragma unroll
            for (int u = 0; u < BATCH; u++) {
                if (c0 + 16 * u < hidden) {
                    const float4 xv = *reinterpret_cast<const float4*>(xr + c0 + 16 * u);
                    acc[0] = fmaf(bf16_lo(wv[u].x), xv.x, acc[0]);
                    acc[1] = fmaf(bf16_hi(wv[u].x), xv.y, acc[1]);
                    acc[2] = fmaf(bf16_lo(wv[u].y), xv.z, acc[2]);
                    acc[3] = fmaf(bf16_hi(wv[u].y), xv.w, acc[3]);
                }
            }
        }
    }
    // acc0 + acc1 lane-wise: lane l of the first accumulator (q = l/4) plus
    // lane l of the second (q = 2 + l/4): the thread two to the right.
    float v[4];
#pragma unroll
    for (int l = 0; l < 4; l++) v[l] = acc[l] + __shfl_xor_sync(0xffffffffu, acc[l], 2);
    // Now q = 0 holds v0..v3 and q = 1 holds v4..v7 (q = 2,3 hold copies).
    // hsum: (v0+v4, v1+v5, v2+v6, v3+v7) -> (s0+s2, s1+s3) -> sum.
    float sv[4];
#pragma unroll
    for (int l = 0; l < 4; l++) sv[l] = v[l] + __shfl_xor_sync(0xffffffffu, v[l], 1);
    const float y = (sv[0] + sv[2]) + (sv[1] + sv[3]);
    // The dot's scalar tail is an empty sum (hidden is a multiple of 32): hsum + 0.0.
    return y + 0.0f;
}

// Router logits of one token, experts e_lo..e_hi-1, into slog[e] (and, when given, their order keys into
// skey[e] and the logits into a global row), by every thread of the CTA, four per expert. `staged`: rows e_lo.. of the router
// matrix in shared memory, or null. The caller puts a CTA barrier after it.
__device__ __forceinline__ void route_logits(const uint16_t* router, const uint8_t* staged, int wstride,
                                             const float* xrow, const float* bias, int hidden, int e_lo, int e_hi,
                                             float* slog, float* logits_row, int tid, int nthreads,
                                             int* skey = nullptr) {
    for (int e0 = e_lo; e0 < e_hi; e0 += nthreads / 4) {
        const int e = e0 + (tid >> 2);
        const bool valid = e < e_hi;
        float y = route_dot_quad(router, staged, wstride, xrow, hidden, valid ? e : e_lo, tid & 3,
                                 e0 + ((tid >> 5) << 3) < e_hi, valid ? e - e_lo : 0);
        if (valid && (tid & 3) == 0) {
            if (bias) y = y + bias[e];
            slog[e] = y;
            if (skey) skey[e] = total_key(y);
            if (logits_row) logits_row[e] = y;
        }
    }
}

// exp(x) for x <= 0 in double precision, rounded to float: what the gating softmax needs
// (its arguments are score - max score). Argument reduction by ln 2 in two parts, a
// degree-13 Taylor polynomial on |r| <= ln(2)/2 (truncation error below 1e-17), and the
// power of two put into the exponent. Results below the smallest float flush to zero as
// the conversion would make them.
__device__ __forceinline__ float exp_nonpositive_f64(float xf) {
    if (xf != xf) return xf;
    if (xf < -104.0f) return 0.0f;
    const double x = double(xf);
    const double n = rint(x * 1.4426950408889634);
    double r = fma(-n, 6.93147180369123816490e-01, x);
    r = fma(-n, 1.90821492927058770002e-10, r);
    double p = 1.0 / 6227020800.0;
    p = fma(p, r, 1.0 / 479001600.0);
    p = fma(p, r, 1.0 / 39916800.0);
    p = fma(p, r, 1.0 / 3628800.0);
    p = fma(p, r, 1.0 / 362880.0);
    p = fma(p, r, 1.0 / 40320.0);
    p = fma(p, r, 1.0 / 5040.0);
    p = fma(p, r, 1.0 / 720.0);
    p = fma(p, r, 1.0 / 120.0);
    p = fma(p, r, 1.0 / 24.0);
    p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    const long long bits = __double_as_longlong(p) + (static_cast<long long>(n) << 52);
    return float(__longlong_as_double(bits));
}

// Top-k and gates of one token, by ONE warp: lane l holds experts l, l+32, .... Up to 64 experts: each
// lane ranks its experts against all keys (written over the logits, which are given up) and the picks are
// scattered to their ranks; above, k rounds of taking the largest. Lane j < k ends with the j-th pick and
// writes ids_row[j] / gates_row[j]. slog is 16-byte aligned and readable up to a multiple of 4 experts.
__device__ __forceinline__ void route_topk_gates(float* slog, int experts, int topk, uint32_t* ids_row,
                                                 float* gates_row, int lane) {
    int my_id = 0;
    float my_val = 0.0f;
    if (experts <= 64) {
        // Larger key first, lower index first among equals: lane's experts `lane` and `lane + 32`.
        int* skey = reinterpret_cast<int*>(slog);
        const bool on0 = lane < experts, on1 = lane + 32 < experts;
        const float val0 = on0 ? slog[lane] : 0.0f, val1 = on1 ? slog[lane + 32] : 0.0f;
        const int key0 = total_key(val0), key1 = total_key(val1);
        __syncwarp();
        if (on0) skey[lane] = key0;
        if (on1) skey[lane + 32] = key1;
        __syncwarp();
        const unsigned below = (1u << lane) - 1u;
        int rank0 = __popc(__match_any_sync(0xffffffffu, key0) & __ballot_sync(0xffffffffu, on0) & below);
        int rank1 = __popc(__match_any_sync(0xffffffffu, key1) & __ballot_sync(0xffffffffu, on1) & below);
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
            if (j < experts) {
                const int4 k4 = *reinterpret_cast<const int4*>(skey + j);
                const int kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (j + i < experts) {
                        rank0 += kk[i] > key0 ? 1 : 0;                           // (equals among 0..31: counted above; 32.. come after)
                        if (experts > 32) rank1 += (j + i < 32 ? kk[i] >= key1 : kk[i] > key1) ? 1 : 0;
                    }
                }
            }
        }
        __syncwarp();
        // The picks to their ranks: ids over the first words, scores behind them (topk <= 32, and the row
        // has experts >= topk words; with fewer than 2 topk words the scores follow in a second step).
        if (on0 && rank0 < topk) skey[rank0] = lane;
        if (on1 && rank1 < topk) skey[rank1] = lane + 32;
        __syncwarp();
        if (lane < topk) my_id = skey[lane];
        __syncwarp();
        if (on0 && rank0 < topk) slog[rank0] = val0;
        if (on1 && rank1 < topk) slog[rank1] = val1;
        __syncwarp();
        if (lane < topk) my_val = slog[lane];
    } else {
        constexpr int SLOTS = MAX_EXPERTS / 32;
        const int nslots = (experts + 31) >> 5;
        unsigned ukeys[SLOTS];  // order-preserving unsigned keys; 0 = not a candidate
        unsigned taken = 0;
    #pragma unroll
        for (int s = 0; s < SLOTS; s++) {
            const int e = lane + 32 * s;
            // total_key is a signed order; flipping the sign bit makes it unsigned. +1 keeps 0 free
            // (the all-ones key, -NaN's neighbour in this order, cannot occur: it would be key 2^32).
            ukeys[s] = (s < nslots && e < experts) ? (unsigned(total_key(slog[e])) ^ 0x80000000u) : 0u;
            if (!(s < nslots && e < experts)) taken |= 1u << s;
        }
        for (int j = 0; j < topk; j++) {
            unsigned best_key = 0;
            int best_idx = 0x7fffffff;
    #pragma unroll
            for (int s = 0; s < SLOTS; s++) {
                if (s < nslots && !((taken >> s) & 1u)) {
                    if (best_idx == 0x7fffffff || ukeys[s] > best_key) {
                        best_key = ukeys[s];
                        best_idx = lane + 32 * s;
                    }
                }
            }
            // The largest key in the warp, then the lowest expert index among its holders.
            const bool have = best_idx != 0x7fffffff;
            const unsigned wmax = __reduce_max_sync(0xffffffffu, have ? best_key : 0u);
            const bool tie = have && best_key == wmax;
            const unsigned widx = __reduce_min_sync(0xffffffffu, tie ? unsigned(best_idx) : 0xffffffffu);
            const int win = int(widx);
            if ((win & 31) == lane) taken |= 1u << (win >> 5);
            if (lane == j) {
                my_id = win;
                my_val = slog[win];
            }
        }
    }
    const float mx = __shfl_sync(0xffffffffu, my_val, 0);
    float ej = 0.0f;
    if (lane < topk) ej = exp_nonpositive_f64(my_val - mx);
    float sum = 0.0f;
    for (int j = 0; j < topk; j++) sum = sum + __shfl_sync(0xffffffffu, ej, j);
    if (lane < topk) {
        ids_row[lane] = uint32_t(my_id);
        gates_row[lane] = __fdiv_rn(ej, sum);
    }
}

// How many of the token's experts come before expert 32 group + lane, whose key is `key` (`on`: there is such an expert).
// Experts of groups before this one come first among equals, those of groups behind it do not; within the
// group the lower lanes do. Whole warps; skey 16-byte aligned and readable up to a multiple of 4 experts.
__device__ __forceinline__ int rank_in_order(const int* skey, int experts, int group, int key, bool on, int lane) {
    int rank = __popc(__match_any_sync(0xffffffffu, key) & __ballot_sync(0xffffffffu, on) & ((1u << lane) - 1u));
#pragma unroll 1
    for (int j0 = 0; j0 < experts; j0 += 32) {
        const bool before = (j0 >> 5) < group;
#pragma unroll
        for (int u = 0; u < 32; u += 4) {
            if (j0 + u < experts) {
                const int4 k = *reinterpret_cast<const int4*>(skey + j0 + u);
                const int kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (j0 + u + i < experts && (before ? kk[i] >= key : kk[i] > key)) rank++;
            }
        }
    }
    return rank;
}

// Top-k of one token by a whole CTA, a thread per expert: each counts the experts that come before its
// own in the order (larger key first, lower index first among equals) by reading all keys, four
// at a time, from shared memory; the thread of rank j < topk has the j-th pick, its id into id_out[j] and
// s_id[j], its score into s_val[j]. The picks of route_topk_gates without a chain of dependent rounds.
// skey[e] = total_key of expert e's logit, 16-byte aligned, readable up to a multiple of 4 experts; the
// caller puts a CTA barrier before and after. Whole warps take part.
__device__ __forceinline__ void route_rank_picks(const int* skey, const float* slog, int experts, int topk,
                                                 uint32_t* id_out, uint32_t* s_id, float* s_val, int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    if (warp * 32 >= experts) return;
    const bool on = tid < experts;
    const int key = on ? skey[tid] : 0;
    const int rank = rank_in_order(skey, experts, warp, key, on, lane);
    if (on && rank < topk) {
        if (id_out) id_out[rank] = uint32_t(tid);
        s_id[rank] = uint32_t(tid);
        s_val[rank] = slog[tid];
    }
}

// The gates of those picks by ONE warp (lane j the j-th): softmax over the scores with the top score
// as the maximum, the sum taken in score order.
__device__ __forceinline__ float route_pick_gate(const float* s_val, int topk, int lane) {
    const float my_val = lane < topk ? s_val[lane] : 0.0f;
    const float mx = __shfl_sync(0xffffffffu, my_val, 0);
    float ej = 0.0f;
    if (lane < topk) ej = exp_nonpositive_f64(my_val - mx);
    float sum = 0.0f;
    for (int j = 0; j < topk; j++) sum = sum + __shfl_sync(0xffffffffu, ej, j);
    return __fdiv_rn(ej, sum);
}

// Eight values of a 32-block as quantize_q8 rounds them (src/kernels.rs:84-98), packed: half away from
// zero (truncation after adding the float below one half with the value's sign: exact for every
// |v| < 2^22), NaN to 0, the packing saturates. Returns their sum in `qsum`.
__device__ __forceinline__ uint2 quantize_eight(const float4& a, const float4& b, float id, int& qsum) {
    auto q4 = [&](const float4& f) {
        auto q = [&](float x) {
            const float v = x * id;
            return __float2int_rz(v + copysignf(0.49999997f, v));
        };
        uint32_t w = 0;
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q(f.w)), "r"(q(f.z)), "r"(0));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q(f.y)), "r"(q(f.x)), "r"(w));
        return w;
    };
    const uint2 w = make_uint2(q4(a), q4(b));
    qsum = __dp4a(int(w.x), 0x01010101, __dp4a(int(w.y), 0x01010101, 0));
    return w;
}

// A 32-block by four neighbouring lanes, eight values each: every lane gets the block's scale and scaled
// sum of quants, and its own eight bytes. All lanes of the warp take part.
__device__ __forceinline__ uint2 quantize_block_quad(const float4& a, const float4& b, float& scale, float& sum) {
    float amax = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                       fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));  // (fmaxf drops NaNs, as f32::max)
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f);
    int qsum;
    const uint2 w = quantize_eight(a, b, d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f, qsum);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
    scale = d;
    sum = d * float(qsum);
    return w;
}

// 8-bit quantization of one token's row (16-byte aligned, in shared memory), four lanes per 32-block: warps
// first_warp .. first_warp + nq - 1 of the CTA take eight blocks at a time (and the zero padding up
// to whole super-blocks of the scale rows).
__device__ __forceinline__ void route_quantize_row(const float* xrow, int hidden, int8_t* xq_row, float* xs_row,
                                                         float* xsum_row, int warp, int lane, int first_warp, int nq) {
    const int nb = hidden / QK;
    const int padded = (nb + SUPER - 1) / SUPER * SUPER;
    for (int b0 = (warp - first_warp) * 8; warp >= first_warp && b0 < padded; b0 += nq * 8) {
        const int b = b0 + (lane >> 2), q = lane & 3;
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        if (b < nb) {
            lo = *reinterpret_cast<const float4*>(xrow + b * QK + q * 8);
            hi = *reinterpret_cast<const float4*>(xrow + b * QK + q * 8 + 4);
        }
        float d, su;
        const uint2 w = quantize_block_quad(lo, hi, d, su);
        if (b < nb) *reinterpret_cast<uint2*>(xq_row + b * QK + q * 8) = w;
        if (b < padded && q == 0) xs_row[b] = d, xsum_row[b] = su;
    }
}

// Rows kept in shared memory with four floats of padding after every 32-element block: lanes that each walk a
// block of their own then spread over the banks, and 16-byte accesses stay aligned.
constexpr int ROW_PAD_BLOCK = QK + 4;

}  // namespace tc
