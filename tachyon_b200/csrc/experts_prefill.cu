// Grouped expert products for prefill-size groups on the 5th-generation tensor
// cores (tcgen05), whose results are scaled and added up block by block on the FP32 pipe.
//
// Arithmetic: the same single fma chain per output as the decode-size kernels
// (experts_fast.cuh), so a token's value does not depend on which kernel ran:
//     acc = fma(float(sum_b), ws[row,b] * xs[token,b], acc)      b = 0, 1, ...
// One block of 32 columns is one product of its own into its own tensor-memory buffer: the block's
// sums must leave the tensor core to be scaled before they can be added.
//
// What bounds it, in cycles per 128 x 64 x 32 unit and SM: that float work, two packed FP32 operations per output pair
// and block, 128 (and 34 of the finishing warps); the reads of tensor memory, 128 (the 16-lane shape moves half of what
// the 32-lane one does) beside the products' own 37; and shared memory at 128 bytes a clock: 64 for the products'
// operands, 66 for the copies that bring them, 80 for the scales (if lanes that read the same word cost as much as lanes
// that do not; the measured 188 a unit, less than the sum, says that they cost less). So:
//  - A lane has 4 rows x 16 tokens (the 16x256b shape), 20 words of scales per 64 outputs. With a row of 64 tokens
//    (32x32b) they were 65 words: 272 cycles of shared memory a unit beside the other 130, in units of 365 to 430.
//  - The float loop's code is 4 blocks long with constant addresses, a barrier test and an arrival per 2 blocks;
//    the finishing code is rolled. (Unrolled as far as 16 KB it cost the float warps 20 % in instruction fetches.)
//  - Products are issued and copies made by converged warps, and an operand stage is free again once its products
//    are done; the scales have a longer ring of their own.
//  - The operands are the 8-bit values as f16 (kind::f16). Products and sums of a block are
//    integers below 2^20, exact in the f32 accumulator, so the sums arrive as floats. With kind::i8
//    every sum costs a conversion besides (238 cycles per unit); with mma.sync, which would leave the
//    sums in registers, conversions and a slower instruction (276).
//  - A finished tile is only parked in shared memory by the float warps; four other warps take it
//    from there while the next tile's chains run: for gate_up SwiGLU, 8-bit quantization per
//    32-block (src/kernels.rs:84-98) and the store in the layout the down product reads, so the
//    SwiGLU rows never visit memory in f32; for down the rows' stores.
// Persistent CTAs (one per SM) walk (token tile, 128-row tile) pairs; both rings run across tile
// boundaries. Roles: warps 0-7 float chains (TMEM lane quadrant = warp % 4, half of the tokens
// = warp / 4: a row's weight scale, a barrier wait and a release are paid once per 64 outputs of a
// lane), warp 8 streams operand chunks of 2 blocks, an elected lane of warp 9 issues the products into a ring
// of two TMEM halves, warps 12-15 finish tiles. An expert's tokens are cut into tiles of 128 and a
// remainder of 128, 64 or 32 columns (4-bit: 64 at most, since each output keeps a second chain).
// Every wait is bounded; TMEM is freed on every path.
//
// Measured (granite-1b-a400m, 4096 tokens, int8; 24, now 20 us of gate_up tile the activations): gate_up 234 -> 183 us, down
// 109 -> 86; 64 experts of 2048 x 1024: 812 -> 615, 383 -> 291; 40 of 1536 x 512 in 4 bits at 2047 tokens: 276 -> 209, 138
// -> 109. A chunk of two blocks takes 750 cycles (188 a unit), a tile 3300 besides, and another 3300 of a scheduler's time go
// to finishing it in gate_up; 4-bit tiles, of 64 columns, take 480 a unit, where shared memory alone is up to 386 (192 the
// scales, counted as above, 96 operands, 98 copies). Tried: 16 float warps of 32 columns (as before or slower), the loop rolled to a
// block (bookkeeping: 342 instructions a unit against 177) or to a chunk (211 / 99 us), pieces of 32 values a
// lane (spills), a block's scales read a block ahead (spills), 4-bit tiles of 128 columns (spills), remainders of 65 to 96
// tokens as 64 + 32 columns (333 tokens 42 + 25 -> 54 + 31 us: a narrow tile costs nearly as much as a wide one), the widest
// tiles first (1 %), polling instead of suspended waits (3 % slower), kind::i8 (conversions: 10 % slower), mma.sync with the
// sums in registers (8 % slower).
#include <algorithm>
#include <type_traits>

#include "dispatch_common.cuh"
#include "experts_common.cuh"
#include "umma.cuh"

namespace tc {

namespace {

constexpr int P_ROWS = 128;             // MMA M
constexpr int P_CHUNK = 2;              // blocks per shared-memory stage, and per hand-over of TMEM buffers
constexpr int P_TBUF = 128;             // columns of a TMEM buffer
constexpr int P_NGRP = 2;               // groups of P_CHUNK buffers: all 512 columns
constexpr int P_A_BLOCK = P_ROWS * 64;  // bytes of one block of weights (f16)
constexpr int P_EW = 8;                 // float warps: 4 TMEM lane quadrants x 2 token halves
constexpr int P_IW = 4;                 // producer, MMA issuer and two warps that make up their warpgroup
constexpr int P_FW = 4;                 // finishing warps
constexpr int P_THREADS = (P_EW + P_IW + P_FW) * 32;
constexpr uint32_t P_SPIN = 1u << 16;
constexpr size_t P_SMEM_LIMIT = 227 * 1024 - 256;  // the kernel also has a few static words
constexpr int P_HSTRIDE = P_ROWS + 4;   // floats per parked token (the pad keeps 16-byte reads conflict-free)

// Registers: 128 a thread at launch (ptxas gives a 512-thread block that many), then split.
constexpr int P_REGS_LAUNCH = 128, P_REGS_FLOAT = 176, P_REGS_ISSUE = 56, P_REGS_FINISH = 104;
static_assert((P_EW * P_REGS_FLOAT + P_IW * P_REGS_ISSUE + P_FW * P_REGS_FINISH) * 32 <= P_THREADS * P_REGS_LAUNCH, "register split");

__host__ __device__ constexpr int prefill_columns(bool q4) { return q4 ? 64 : 128; }  // the largest token tile

// Shared memory: a ring of N operand stages (P_CHUNK blocks of weights and activations), left as soon as their products are
// done, a ring of SN sets of their scales, read until the float warps are through with the sums, and a parked tile.
// (Scales in the operands' stages held those back by a chunk, and the copies' latency showed: 4-bit tiles waited 370 of the
// 980 cycles of a chunk for operands.)
template <bool Q4>
struct Stage {
    static constexpr int TOK = prefill_columns(Q4);
    static constexpr int B = P_CHUNK * P_A_BLOCK;
    static constexpr int BYTES = B + P_CHUNK * TOK * 64;
    static constexpr int N = 4;                             // operand stages
    static constexpr int XS = P_CHUNK * P_ROWS * 4;         // (the weights' scales come first)
    static constexpr int WC = XS + P_CHUNK * TOK * 4;       // (4-bit only from here)
    static constexpr int XSUM = WC + P_CHUNK * P_ROWS * 4;
    static constexpr int SET = Q4 ? XSUM + P_CHUNK * TOK * 4 : WC;
    // Sets of scales. Chunk c's go in when the products of chunk c - N are done, and those waited for the float warps to be
    // through with chunk c - N - P_NGRP.
    static constexpr int SN = 8;
    static_assert(SN >= N + P_NGRP, "a set is read before it is overwritten");
    static constexpr int PARK = TOK * P_HSTRIDE * 4;
    static constexpr int SCALES = N * BYTES, PARKED = SCALES + SN * SET, BARS = PARKED + PARK;
    static constexpr size_t SMEM = size_t(BARS) + (2 * N + 2 * P_NGRP + 3) * 8;
    static_assert(SMEM <= P_SMEM_LIMIT, "stages fit");
};

using umma::f16_tile_offset;

struct PrefillArgs {
    const uint16_t* wt;      // weight tiles, f16 [expert][row tile][block][128 x 32 canonical]
    const float* wd;         // weight block scales [expert][row tile][nb][128]
    const float* wc;         // 4-bit block offsets, same shape (null for 8-bit)
    const uint16_t* xt;      // activation tiles, f16: tile at row0 * 32 * nb, [block][N x 32 canonical]
    const float* xst;        // activation scales: tile at row0 * nb, [block][N]
    const float* xsumt;      // scale * sum of quants, same shape (4-bit only)
    const TokenTile* tiles;
    const int* tile_count;
    int nb, row_tiles, out_cols;
    // gate_up: the SwiGLU rows as the down product's activation tiles (nb_out = out_cols / 32 blocks)
    uint16_t* xt_out;
    float* xst_out;
    float* xsumt_out;
    // down: rows of f32
    float* out;
    const uint32_t* out_rows;
    float one;               // 1.0f, a value the compiler does not know (see add2_exact)
    int* status;
};

// Expert parallel (down only): row p of out_rows' numbering belongs to rank p / rows and goes
// straight into that rank's window, at row p % rows. (A kernel argument of its own: with these
// fields inside PrefillArgs the kernels that do not use them ran 9 % slower.)
struct PrefillPeer {
    float* out[MAX_PEERS];
    uint32_t rows;
    int ranks;
};
struct NoPeer {};

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait. One that runs out sets the CTA's abort flag, and every wait after that gives up at
// once; the warps then run on to the end over whatever they find (every address they form stays in
// bounds) and the kernel reports the failure. Waits that could leave the loops instead would make
// every loop counter, and with it every address, a per-lane value to the compiler: each tensor
// memory load would then wait for a move into a uniform register.
__device__ __forceinline__ void wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_test(bar, parity)) return;
    for (uint32_t i = 0; i < P_SPIN; i++)
        if (mbar_try_wait(bar, parity) || *abort_flag) return;
    *abort_flag = 1;
}

__device__ __forceinline__ void mbar_arrive_if(uint64_t* bar, bool mine) {  // predicated: no branch around it
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(
                     smem_addr(bar)),
                 "r"(uint32_t(mine))
                 : "memory");
}

// The same value in every lane, told to the compiler.
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }

// Four signed bytes as f16: 1024 + (v + 128) is exact in f16 and is v + 1152.
__device__ __forceinline__ uint2 f16_from_s8(uint32_t w) {
    const uint32_t u = w ^ 0x80808080u;
    const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
    uint32_t lo = __byte_perm(u, 0x64646464u, 0x4140), hi = __byte_perm(u, 0x64646464u, 0x4342);
    const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo), bias), h = __hsub2(*reinterpret_cast<__half2*>(&hi), bias);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}

// A role's place in the rings is one number, the chunks of the CTA's sequence so far, across tiles:
// chunk c is in operand stage c % 4, scale set c % 8 and TMEM half c % 2.
template <bool Q4>
__device__ __forceinline__ uint32_t stage_of(uint32_t c) { return c % Stage<Q4>::N; }
template <bool Q4>
__device__ __forceinline__ uint32_t stage_par(uint32_t c) { return (c / Stage<Q4>::N) & 1; }
__device__ __forceinline__ uint32_t half_of(uint32_t c) { return c % P_NGRP; }
__device__ __forceinline__ uint32_t half_par(uint32_t c) { return (c / P_NGRP) & 1; }

struct Bars {
    uint64_t *full, *empty;    // [stages] operands and scales landed; left by the MMAs
    uint64_t *tfull, *tempty;  // [P_NGRP] a chunk's sums are in TMEM, its scales in shared memory; read by every float warp
    uint64_t *pfull, *pempty;  // a tile has been parked by every float warp; taken by every finishing warp
    uint64_t* drain;           // after a failure only: the issuer's MMAs so far are done
    volatile int* abort_flag;
};

// The token tile of a CTA's work item, read one item ahead by every role: the trip to L2 would otherwise stand at the
// start of each tile, in every warp.
__device__ __forceinline__ TokenTile tile_of(const PrefillArgs& a, int w, int work) {
    return a.tiles[w < work ? w / a.row_tiles : 0];
}

__device__ __forceinline__ float4 staged_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 staged_f2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
// Where a tile's logical row sits in the product, so that a lane's four rows are neighbours (see float_chains).
__host__ __device__ constexpr int product_row(int r) { return (r & ~31) + (r & 3) * 8 + ((r & 31) >> 2); }
// Where a token's scale sits among its tile's: a lane's four columns of every sixteen are neighbours.
__host__ __device__ constexpr int scale_place(int n) { return (n & ~15) + ((n & 7) >> 1) * 4 + ((n & 8) >> 2) + (n & 1); }

// One tile's float work for this warp's 32 rows x CW tokens: reads each block's sums from TMEM half a block (the lower
// or upper 16 rows) ahead of the arithmetic (the load is asynchronous until wait_ld, and two register pieces
// alternate) and keeps the chains in registers. A lane has 4 rows x CW / 4 tokens (the order of an m16n8
// accumulator in each half of the quadrant), so a block's scales are CW / 4 + 4 values a lane; the next block's
// replace them as they are used up. Four blocks, one turn of the TMEM halves, are a pass of the loop: its addresses are
// constants but for the stages', and a chunk costs one test of a barrier and one arrival. `turn`: turns so far.
template <bool Q4, int CW>
__device__ __forceinline__ void float_chains(float (&acc)[64], float (&off)[Q4 ? 32 : 1], uint32_t& turn, uint32_t smem,
                                             const Bars& bars, uint32_t tbase, int nb, int col0, int row0, int lane) {
    using S = Stage<Q4>;
    // A piece: half of the rows x up to 32 columns.
    constexpr int N = CW * 2, CC = CW < 32 ? CW : 32, PC = CC / 2, PIECES = CW / CC * 2;
    float v[2][PC];
    float2 w[2], wc[Q4 ? 2 : 1];
    float4 x[CW / 16], u[Q4 ? CW / 16 : 1];
    const uint32_t wat = S::SCALES + (row0 + (lane >> 2) * 4) * 4, xat = S::SCALES + S::XS + (col0 + (lane & 3) * 4) * 4;
    auto row_scales = [&](uint32_t st, int k, int h) {  // of the lane's two rows in half h
        w[h] = staged_f2(st + wat + (k * P_ROWS + 2 * h) * 4);
        if (Q4) wc[Q4 ? h : 0] = staged_f2(st + wat + S::WC + (k * P_ROWS + 2 * h) * 4);
    };
    auto column_scales = [&](uint32_t st, int k, int j) {  // of the lane's columns among sixteen
        x[j] = staged_f4(st + xat + (k * N + j * 16) * 4);
        if (Q4) u[Q4 ? j : 0] = staged_f4(st + xat + (S::XSUM - S::XS) + (k * N + j * 16) * 4);
    };
    auto chains = [&](const float (&cur)[PC], int p, int j) {  // columns 16 j .. of piece p
        const int h = p & 1;
        const float w2[2] = {w[h].x, w[h].y}, c2[2] = {wc[Q4 ? h : 0].x, wc[Q4 ? h : 0].y};
        const float4 xj = x[j], uj = u[Q4 ? j : 0];
#pragma unroll
        for (int q = 0; q < 2; q++) {  // 8 columns: two rows x two neighbouring tokens
            const float2 x2 = q ? make_float2(xj.z, xj.w) : make_float2(xj.x, xj.y);
            const float2 u2 = q ? make_float2(uj.z, uj.w) : make_float2(uj.x, uj.y);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int i = 8 * (j - p / 2 * (CC / 16)) + 4 * q + 2 * r, o = p * PC + i;
                const float2 s = fma2(make_float2(cur[i], cur[i + 1]), mul2(splat(w2[r]), x2), make_float2(acc[o], acc[o + 1]));
                acc[o] = s.x, acc[o + 1] = s.y;
                if (Q4) {
                    const float2 f = fma2(splat(c2[r]), u2, make_float2(off[o], off[o + 1]));
                    off[o] = f.x, off[o + 1] = f.y;
                }
            }
        }
    };
#pragma unroll
    for (int j = 0; j < CW; j++) {
        acc[j] = 0.0f;
        if (Q4) off[j] = 0.0f;
    }
    const uint32_t sums = tbase + col0;
    auto set_of = [](uint32_t turn) { return turn % (S::SN / P_NGRP) * P_NGRP; };  // a turn's first set of scales
    auto fetch = [&](uint32_t at, int p) { umma::ld_half_f32(at + p / 2 * 32 + (uint32_t(p & 1) << 20), v[p & 1]); };
    auto first_scales = [&](uint32_t st, int k) {
        row_scales(st, k, 0);
        row_scales(st, k, 1);
#pragma unroll
        for (int j = 0; j < CW / 16; j++) column_scales(st, k, j);
    };
    // A half's chunk has been read, sums and scales: the issuer may overwrite them.
    auto release = [&](int half) {
        umma::fence_before_sync();
        __syncwarp();
        mbar_arrive_if(bars.tempty + half, lane == 0);
    };
    const int whole = nb / (P_NGRP * P_CHUNK);
    if (whole > 0) {
        wait_or_abort(bars.tfull, turn & 1, bars.abort_flag);
        umma::fence_after_sync();
        fetch(sums, 0);
        first_scales(smem + set_of(turn) * S::SET, 0);
    }
#pragma unroll 1
    for (int t = 1; t <= whole; t++, turn++) {
        const uint32_t par = turn & 1, st = smem + set_of(turn) * S::SET, other = smem + set_of(turn + 1) * S::SET;
        const bool again = t < whole;
#pragma unroll
        for (int i = 0; i < P_NGRP * P_CHUNK; i++) {
            const int half = i / P_CHUNK, kn = (i + 1) % P_CHUNK;
            const bool ends = kn == 0, last = i + 1 == P_NGRP * P_CHUNK, more = !last || again;
            const uint32_t next = last ? other : st + (i + 1) / P_CHUNK * S::SET;  // where the next block's scales are
            bool ready = true;
#pragma unroll
            for (int p = 0; p < PIECES; p++) {
                const bool final = p + 1 == PIECES;
                umma::wait_ld(v[p & 1]);
                if (final && ends) release(half);
                if (final && ends && more) {
                    if (!ready) wait_or_abort(bars.tfull + (half ^ 1), last ? par ^ 1 : par, bars.abort_flag);
                    umma::fence_after_sync();
                }
                if (!final) fetch(sums + i * P_TBUF, p + 1);
                else if (more) fetch(sums + (last ? 0 : i + 1) * P_TBUF, 0);
                if (p + 2 == PIECES && ends && more) ready = mbar_test(bars.tfull + (half ^ 1), last ? par ^ 1 : par);
                // The next block's scales, as this one's are used up (another chunk's once it is known to be there).
                if (final && ends && more) {
                    row_scales(next, kn, 0);
#pragma unroll
                    for (int j = 0; j < p / 2 * (CC / 16); j++) column_scales(next, kn, j);
                }
#pragma unroll
                for (int j = p / 2 * (CC / 16); j < (p / 2 + 1) * (CC / 16); j++) {
                    chains(v[p & 1], p, j);
                    if ((p & 1) && more && (final || !ends)) column_scales(next, kn, j);
                }
                if (p + 2 == PIECES && !ends) row_scales(next, kn, 0);
                if (final && more) row_scales(next, kn, 1);
            }
        }
    }
    // What is left of a number of blocks that is no multiple of four (a turn all the same, of fewer blocks).
    if (const int rest = nb - whole * P_NGRP * P_CHUNK) {
        const uint32_t st = smem + set_of(turn) * S::SET;
#pragma unroll 1
        for (int half = 0; half < P_NGRP; half++) {
            wait_or_abort(bars.tfull + half, turn & 1, bars.abort_flag);
            umma::fence_after_sync();
#pragma unroll 1
            for (int k = 0; k < P_CHUNK && half * P_CHUNK + k < rest; k++) {
                first_scales(st + half * S::SET, k);
#pragma unroll
                for (int p = 0; p < PIECES; p++) {
                    fetch(sums + (half * P_CHUNK + k) * P_TBUF, p);
                    umma::wait_ld(v[p & 1]);
#pragma unroll
                    for (int j = p / 2 * (CC / 16); j < (p / 2 + 1) * (CC / 16); j++) chains(v[p & 1], p, j);
                }
            }
            release(half);
        }
        turn++;
    }
}

// silu(gate) * up of 32 hidden columns of one token (the parked row holds gate and up side by side),
// then quantize_q8 (src/kernels.rs:84-98) of that block, as f16 into the token's row of the tile. The products go back
// over the gates and ups on the way, and both loops stay short: a straight run of all 32 columns is 16 KB of
// instructions, fetched past the float warps' own.
__device__ __forceinline__ void finish_block(float4* parked, float2 one, uint8_t* dst, int N, float& scale, float& sum) {
    float amax = 0.0f;
#pragma unroll 1
    for (int i = 0; i < 4; i++) {  // 8 columns
        float4 v[4];
        float2 h[4];
        bool usable = true;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = parked[4 * i + j];  // gate, up, gate, up
            h[j] = mul2(silu2(make_float2(v[j].x, v[j].z), one, usable), make_float2(v[j].y, v[j].w));
        }
        if (!usable) {  // (one test for the lot: a branch at every pair would keep them from overlapping)
#pragma unroll 1
            for (int j = 0; j < 4; j++) {
                const float4 u = parked[4 * i + j];
                const float2 t = make_float2(__fdiv_rn(u.x, 1.0f + exp_poly(-u.x)) * u.y, __fdiv_rn(u.z, 1.0f + exp_poly(-u.z)) * u.w);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k == j) h[k] = t;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) amax = fmaxf(fmaxf(amax, fabsf(h[j].x)), fabsf(h[j].y));
        parked[2 * i] = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
        parked[2 * i + 1] = make_float4(h[2].x, h[2].y, h[3].x, h[3].y);
    }
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    int qsum = 0;
#pragma unroll 1
    for (int i = 0; i < 4; i++) {  // 8 columns: 16 bytes of f16
        uint2 f[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            // Rounds half away from zero as exp_poly2 does; NaN becomes 0; the packing saturates.
            const float4 h = parked[2 * i + u];
            int q[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float2 t = mul2(k ? make_float2(h.z, h.w) : make_float2(h.x, h.y), make_float2(id, id));
                q[2 * k] = __float2int_rz(t.x + copysignf(0.49999997f, t.x));
                q[2 * k + 1] = __float2int_rz(t.y + copysignf(0.49999997f, t.y));
            }
            uint32_t w = 0;
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q[3]), "r"(q[2]), "r"(0));
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q[1]), "r"(q[0]), "r"(w));
            qsum = __dp4a(int(w), 0x01010101, qsum);
            f[u] = f16_from_s8(w);
        }
        *reinterpret_cast<uint4*>(dst + i * N * 16) = make_uint4(f[0].x, f[0].y, f[1].x, f[1].y);
    }
    scale = d;
    sum = d * float(qsum);
}

template <bool Q4, bool GATE_UP, bool PEER = false>
__global__ void __launch_bounds__(P_THREADS, 1)
    expert_prefill_kernel(const PrefillArgs a, const std::conditional_t<PEER, PrefillPeer, NoPeer> peer) {
    using S = Stage<Q4>;
    extern __shared__ __align__(128) uint8_t smem[];
    float* parked = reinterpret_cast<float*>(smem + S::PARKED);  // [tokens][P_HSTRIDE] a finished tile
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    Bars bars;
    bars.full = reinterpret_cast<uint64_t*>(smem + S::BARS);
    bars.empty = bars.full + S::N;
    bars.tfull = bars.empty + S::N;
    bars.tempty = bars.tfull + P_NGRP;
    bars.pfull = bars.tempty + P_NGRP;
    bars.pempty = bars.pfull + 1;
    bars.drain = bars.pempty + 1;
    bars.abort_flag = &s_abort;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = int(warp_uniform(uint32_t(tid) >> 5));
    grid_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < S::N; s++) {
            mbar_init(bars.full + s, 1);
            mbar_init(bars.empty + s, 1);
        }
        for (int g = 0; g < P_NGRP; g++) {
            mbar_init(bars.tfull + g, 2);
            mbar_init(bars.tempty + g, P_EW);
        }
        mbar_init(bars.pfull, P_EW);
        mbar_init(bars.pempty, P_FW);
        mbar_init(bars.drain, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == P_EW + 1) {
        umma::tmem_alloc(&s_tmem, P_NGRP * P_CHUNK * P_TBUF);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem;
    grid_dependency_wait();  // everything below reads what earlier kernels wrote
    const int nb = a.nb, turn_blocks = (nb + P_NGRP * P_CHUNK - 1) / (P_NGRP * P_CHUNK) * (P_NGRP * P_CHUNK);
    const int work = int(warp_uniform(uint32_t(*a.tile_count * a.row_tiles)));
    if (warp < P_EW) {
        // ---- float warps
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P_REGS_FLOAT));
        const int quad = warp & 3, slice = warp >> 2;
        const uint32_t tbase = tmem + (uint32_t(quad * 32) << 16);
        uint32_t c = 0;  // turns of the TMEM halves
        uint32_t parity = 1;  // of pempty: the first tile finds the parking space free
        TokenTile ahead = tile_of(a, blockIdx.x, work);
        for (int w = blockIdx.x; w < work; w += gridDim.x) {
            const int N = int(warp_uniform(ahead.cols));
            ahead = tile_of(a, w + gridDim.x, work);
            const int col0 = slice * (N / 2);  // this warp's first token of the tile
            float acc[64], off[Q4 ? 32 : 1];
            if (!Q4 && N == 128) float_chains<Q4, Q4 ? 32 : 64>(acc, off, c, smem_addr(smem), bars, tbase, nb, col0, quad * 32, lane);
            else if (N == 64) float_chains<Q4, 32>(acc, off, c, smem_addr(smem), bars, tbase, nb, col0, quad * 32, lane);
            else float_chains<Q4, 16>(acc, off, c, smem_addr(smem), bars, tbase, nb, col0, quad * 32, lane);
            wait_or_abort(bars.pempty, parity, bars.abort_flag);
            parity ^= 1;
            // A lane's four rows of a token side by side (the 132-float stride spreads the lanes over the banks).
            float* dst = parked + (col0 + 2 * (lane & 3)) * P_HSTRIDE + quad * 32 + (lane >> 2) * 4;
            auto value = [&](int i) { return Q4 ? acc[i] + off[Q4 ? i : 0] : acc[i]; };
            auto park = [&](auto cw) {
                constexpr int CW = decltype(cw)::value, CC = CW < 32 ? CW : 32, H = CC / 2;  // (the order of float_chains)
#pragma unroll
                for (int j = 0; j < CW / 8; j++)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int lo = j / (CC / 8) * CC + j % (CC / 8) * 4 + i;
                        *reinterpret_cast<float4*>(dst + (8 * j + i) * P_HSTRIDE) =
                            make_float4(value(lo), value(lo + 2), value(H + lo), value(H + lo + 2));
                    }
            };
            if (!Q4 && N == 128) park(std::integral_constant<int, Q4 ? 32 : 64>{});
            else if (N == 64) park(std::integral_constant<int, 32>{});
            else park(std::integral_constant<int, 16>{});
            __syncwarp();
            mbar_arrive_if(bars.pfull, lane == 0);
        }
    } else if (warp < P_EW + P_IW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P_REGS_ISSUE));
        // (Both warps run converged, a lane elected for what only one may do: addresses and descriptors then stay in
        // uniform registers. By a lone lane the four products and commit of a chunk took 465 cycles of issue, a
        // chunk 780 of this warp's 1060.)
        if (warp == P_EW) {
            // ---- producer: operand chunks, each once its stage is free again
            asm volatile("fence.proxy.async;" ::: "memory");  // the tiles were written by plain stores
            uint32_t c = 0;
            TokenTile ahead = tile_of(a, blockIdx.x, work);
            for (int w = blockIdx.x; w < work; w += gridDim.x) {
                const uint32_t N = warp_uniform(ahead.cols), expert = warp_uniform(uint32_t(ahead.expert)), row0 = warp_uniform(ahead.row0);
                ahead = tile_of(a, w + gridDim.x, work);
                const size_t wo = (size_t(expert) * a.row_tiles + w % a.row_tiles) * nb, xo = size_t(row0) * nb;
                const uint8_t* wt = reinterpret_cast<const uint8_t*>(a.wt) + wo * P_A_BLOCK;
                const uint8_t* xt = reinterpret_cast<const uint8_t*>(a.xt) + xo * 64;
                const float* wd = a.wd + wo * P_ROWS;
                const float* wc = Q4 ? a.wc + wo * P_ROWS : nullptr;
                const float* xst = a.xst + xo;
                const float* xsumt = Q4 ? a.xsumt + xo : nullptr;
                for (int b0 = 0; b0 < turn_blocks; b0 += P_CHUNK, c++) {
                    const uint32_t nblk = uint32_t(max(0, min(P_CHUNK, nb - b0)));  // (none in the chunks that fill up a turn)
                    uint64_t* full = bars.full + stage_of<Q4>(c);
                    if (c >= uint32_t(S::N)) wait_or_abort(bars.empty + stage_of<Q4>(c), stage_par<Q4>(c) ^ 1, bars.abort_flag);
                    uint8_t* st = smem + stage_of<Q4>(c) * S::BYTES;
                    uint8_t* sc = smem + S::SCALES + c % S::SN * S::SET;
                    const uint32_t wb = nblk * P_A_BLOCK, xb = nblk * N * 64, wf = nblk * P_ROWS * 4, xf = nblk * N * 4;
                    if (umma::elect_one()) {
                        mbar_expect_tx(full, wb + xb + (wf + xf) * (Q4 ? 2 : 1));
                        if (nblk) {
                            bulk_copy(st, wt, wb, full);
                            bulk_copy(st + S::B, xt, xb, full);
                            bulk_copy(sc, wd, wf, full);
                            bulk_copy(sc + S::XS, xst, xf, full);
                            if (Q4) {
                                bulk_copy(sc + S::WC, wc, wf, full);
                                bulk_copy(sc + S::XSUM, xsumt, xf, full);
                            }
                        }
                    }
                    __syncwarp();
                    wt += P_CHUNK * P_A_BLOCK, xt += P_CHUNK * N * 64, wd += P_CHUNK * P_ROWS, xst += P_CHUNK * N;
                    if (Q4) wc += P_CHUNK * P_ROWS, xsumt += P_CHUNK * N;
                }
            }
            if (s_abort) {
                // Giving up: let the copies already issued land before the CTA's shared memory is released.
                for (uint32_t i = c > uint32_t(S::N) ? c - S::N : 0; i < c; i++)
                    mbar_wait_bounded(bars.full + stage_of<Q4>(i), stage_par<Q4>(i));
            }
        } else if (warp == P_EW + 1) {
            // ---- MMA issuer: a block = two K = 16 products into its own TMEM buffer, a commit per chunk
            const uint32_t sums = warp_uniform(tmem);
            uint32_t c = 0;
            TokenTile ahead = tile_of(a, blockIdx.x, work);
            for (int w = blockIdx.x; w < work; w += gridDim.x) {
                const uint32_t N = warp_uniform(ahead.cols), idesc = umma::idesc_f16(P_ROWS, int(N));
                ahead = tile_of(a, w + gridDim.x, work);
                for (int b0 = 0; b0 < turn_blocks; b0 += P_CHUNK, c++) {
                    const int nblk = nb - b0;
                    wait_or_abort(bars.full + stage_of<Q4>(c), stage_par<Q4>(c), bars.abort_flag);
                    if (c >= uint32_t(P_NGRP)) wait_or_abort(bars.tempty + half_of(c), half_par(c) ^ 1, bars.abort_flag);
                    umma::fence_after_sync();
                    // (Low words of the descriptors: address and K stride; the rest is the same for all.)
                    const uint32_t sa = smem_addr(smem + stage_of<Q4>(c) * S::BYTES), sb = sa + S::B;
                    const uint32_t da = umma::smem_desc_low(sa, P_ROWS * 16), db = umma::smem_desc_low(sb, N * 16);
                    const uint32_t d = sums + half_of(c) * P_CHUNK * P_TBUF;
                    if (umma::elect_one()) {
#pragma unroll
                        for (int k = 0; k < P_CHUNK; k++) {
                            if (k < nblk) {
#pragma unroll
                                for (int h = 0; h < 2; h++)
                                    umma::mma_f16_low(d + k * P_TBUF, da + (k * P_A_BLOCK + h * P_ROWS * 32) / 16, db + (k * 2 + h) * N * 2, idesc, uint32_t(h));
                            }
                        }
                        umma::commit(bars.tfull + half_of(c));
                        mbar_arrive_if(bars.tfull + half_of(c), true);  // (what this warp saw land, the float warps may read)
                        umma::commit(bars.empty + stage_of<Q4>(c));
                    }
                    __syncwarp();
                }
            }
            if (s_abort) {
                // Giving up: the MMAs in flight must finish before TMEM is freed.
                if (umma::elect_one()) umma::commit(bars.drain);
                __syncwarp();
                mbar_wait_bounded(bars.drain, 0);
            }
        }
    } else {
        // ---- finishing warps
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P_REGS_FINISH));
        const int ftid = tid - (P_EW + P_IW) * 32;
        const float2 one = make_float2(a.one, a.one);
        uint32_t parity = 0;  // of pfull
        TokenTile ahead = tile_of(a, blockIdx.x, work);
        for (int w = blockIdx.x; w < work; w += gridDim.x, parity ^= 1) {
            const TokenTile tile = ahead;
            ahead = tile_of(a, w + gridDim.x, work);
            const int rt = w % a.row_tiles, N = int(tile.cols), tile_n = int(tile.n);
            wait_or_abort(bars.pfull, parity, bars.abort_flag);
            if (GATE_UP) {
                // A thread per (token, 32-block of hidden columns). Padding tokens are left as they are:
                // their columns are never stored.
                const int nb_out = a.out_cols / QK;
#pragma unroll 1
                for (int i = ftid; i < N * 2; i += P_FW * 32) {
                    const int n = i & (N - 1), q = i / N, b = rt * 2 + q;
                    if (n >= tile_n || b >= nb_out) continue;
                    uint8_t* dst = reinterpret_cast<uint8_t*>(a.xt_out + size_t(tile.row0) * a.out_cols + size_t(b) * N * 32) +
                                   f16_tile_offset(N, n, 0);
                    float d, su;
                    finish_block(reinterpret_cast<float4*>(parked + n * P_HSTRIDE + q * 64), one, dst, N, d, su);
                    const size_t so = size_t(tile.row0) * nb_out + size_t(b) * N + scale_place(n);
                    a.xst_out[so] = d;
                    a.xsumt_out[so] = su;
                }
            } else {
                // A warp per token row, 16 bytes a lane. (out_cols is a multiple of 32.)
                const int r = rt * P_ROWS + lane * 4;
#pragma unroll 4
                for (int n = ftid >> 5; n < tile_n; n += P_FW) {
                    const float4 v = *reinterpret_cast<const float4*>(parked + n * P_HSTRIDE + lane * 4);
                    size_t p = tile.p0 + n;
                    if (a.out_rows) p = a.out_rows[p];
                    float* dst = a.out;
                    if constexpr (PEER) {
                        const uint32_t home = uint32_t(p) / peer.rows;
                        p -= size_t(home) * peer.rows;
                        dst = peer.out[home];
                    }
                    if (r < a.out_cols) *reinterpret_cast<float4*>(dst + p * a.out_cols + r) = v;
                }
            }
            __syncwarp();
            mbar_arrive_if(bars.pempty, lane == 0);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == P_EW + 1) umma::tmem_dealloc(tmem, P_NGRP * P_CHUNK * P_TBUF);
    if (tid == 0 && s_abort) atomicExch(a.status, ERR_COPY_WAIT_TIMEOUT);
}

// ---------------------------------------------------------------- tiling kernels

// Weights as f16 into canonical 128 x 32 tiles per block, with their block scales (and 4-bit offsets) as
// f32 per (block, row); gate_up rows interleaved (gate, up, gate, ...). 4-bit values become q - 8. A
// thread per (row, block), a warp's lanes on 32 consecutive rows: 32-byte reads, 512-byte runs of stores.
// blockIdx.y: a range of P_WT_BLOCKS blocks.
constexpr int P_WT_BLOCKS = 8;
template <bool Q4, bool GATE_UP>
__global__ void __launch_bounds__(256)
    tile_prefill_weights_kernel(const uint8_t* __restrict__ wdata, const void* __restrict__ wscales, int cols,
                                int rows_per_expert, int row_tiles, uint16_t* __restrict__ wt, float* __restrict__ wd,
                                float* __restrict__ wc) {
    const int rt = blockIdx.x % row_tiles, e = blockIdx.x / row_tiles;
    const int nb = cols / QK;
    const int b_lo = blockIdx.y * P_WT_BLOCKS, b_n = min(P_WT_BLOCKS, nb - b_lo);
    for (int task = threadIdx.x; task < P_ROWS * b_n; task += 256) {
        const int r = task % P_ROWS, b = b_lo + task / P_ROWS;
        int row;
        if (GATE_UP) {
            const int inter = rows_per_expert / 2, col = rt * 64 + (r >> 1);
            row = col < inter ? e * rows_per_expert + (r & 1 ? inter : 0) + col : -1;
        } else {
            const int rr = rt * P_ROWS + r;
            row = rr < rows_per_expert ? e * rows_per_expert + rr : -1;
        }
        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // the block's 32 values as signed bytes
        float d = 0.0f, c = 0.0f;
        if (row >= 0) {
            if (!Q4) {
                const uint4* src = reinterpret_cast<const uint4*>(wdata + size_t(row) * cols + b * QK);
                const uint4 lo = src[0], hi = src[1];
                w[0] = lo.x, w[1] = lo.y, w[2] = lo.z, w[3] = lo.w;
                w[4] = hi.x, w[5] = hi.y, w[6] = hi.z, w[7] = hi.w;
                d = f16_bits_to_f32(reinterpret_cast<const uint16_t*>(wscales)[size_t(row) * nb + b]);
            } else {
                // Low nibbles are elements 0..15, high nibbles 16..31.
                const uint4 v = *reinterpret_cast<const uint4*>(wdata + (size_t(row) * cols) / 2 + b * 16);
                const uint32_t n[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    w[i] = uint32_t(nibbles_minus8(n[i] & 0x0F0F0F0Fu));
                    w[4 + i] = uint32_t(nibbles_minus8((n[i] >> 4) & 0x0F0F0F0Fu));
                }
                const int words = (nb + SUPER - 1) / SUPER * SUPER_WORDS;
                const uint32_t* sw = reinterpret_cast<const uint32_t*>(wscales) + size_t(row) * words + (b / SUPER) * SUPER_WORDS;
                const int j = b % SUPER;
                d = f16_bits_to_f32(uint16_t(sw[0])) * float((sw[1 + j / 4] >> (8 * (j % 4))) & 0xFFu);
                c = f16_bits_to_f32(uint16_t(sw[0] >> 16)) * float(int(int8_t(uint8_t(sw[3 + j / 4] >> (8 * (j % 4))))));
            }
        }
        const size_t at = (size_t(e) * row_tiles + rt) * nb + b;
        uint8_t* dst = reinterpret_cast<uint8_t*>(wt) + at * P_A_BLOCK + f16_tile_offset(P_ROWS, product_row(r), 0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint2 f0 = f16_from_s8(w[2 * i]), f1 = f16_from_s8(w[2 * i + 1]);
            *reinterpret_cast<uint4*>(dst + i * P_ROWS * 16) = make_uint4(f0.x, f0.y, f1.x, f1.y);
        }
        wd[at * P_ROWS + r] = d;
        if (Q4) wc[at * P_ROWS + r] = c;
    }
}

// (A dispatch that was given the tile list has built it already.)
__global__ void __launch_bounds__(MAX_EXPERTS)
    build_token_tiles_kernel(const uint32_t* counts, const uint32_t* offsets, int experts, int most_cols,
                             TokenTile* tiles, int* tile_count) {
    __shared__ int s_tiles[MAX_EXPERTS / 32], s_rows[MAX_EXPERTS / 32];
    grid_launch_dependents();
    grid_dependency_wait();
    token_tiles_body(counts, offsets, experts, most_cols, tiles, tile_count, s_tiles, s_rows);
}

// The 8-bit rows of the block's input (xq/xs/xsum through row_of_slot) as f16 into canonical
// (columns x 32) tiles per (token tile, block), scales (and block sums) transposed to
// [block][token]. blockIdx.y: a range of P_ACT_BLOCKS blocks. Padding tokens are left as they are.
// A warp takes 8 tokens x 4 blocks, a lane one of each: its reads and stores then touch 4 to 8 lines an instruction, and the
// rows of both its tasks are asked for before the first is used. Bound by those reads (without them 11 us of the 20, without
// the stores 18). (With 32 tokens of one block a warp every read was 32 lines: 4096 tokens of the 1b shape 24 us, now 20;
// of 2048 columns 39, now 31. Four tasks a thread: 24, for the registers.)
constexpr int P_ACT_BLOCKS = 4, P_ACT_TASKS = 2;  // (128 / 8 token groups over 8 warps)
template <bool Q4>
__global__ void __launch_bounds__(256)
    tile_activations_kernel(const int8_t* xq, const float* xs, const float* xsum, const uint32_t* row_of_slot, int cols,
                            int nbp, const TokenTile* tiles, const int* tile_count, uint16_t* xt, float* xst, float* xsumt) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int nb = cols / QK;
    const int count = *tile_count;
    const TokenTile tile = tiles[blockIdx.x];  // (asked for beside the count: what is past it is left unread)
    if (int(blockIdx.x) >= count) return;
    const int N = tile.cols, b_lo = blockIdx.y * P_ACT_BLOCKS, b_n = min(P_ACT_BLOCKS, nb - b_lo);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, groups = N / 8, tasks = groups * ((b_n + 3) / 4);
    int n[P_ACT_TASKS], b[P_ACT_TASKS];
    bool on[P_ACT_TASKS];
    size_t row[P_ACT_TASKS];
#pragma unroll
    for (int i = 0; i < P_ACT_TASKS; i++) {
        const int task = warp + 8 * i;
        n[i] = (task & (groups - 1)) * 8 + (lane & 7);
        b[i] = b_lo + task / groups * 4 + (lane >> 3);
        on[i] = task < tasks && n[i] < tile.n && b[i] < b_lo + b_n;
        row[i] = on[i] ? row_of_slot[tile.p0 + n[i]] : 0;
    }
    uint4 in[P_ACT_TASKS][2];
    float d[P_ACT_TASKS], su[Q4 ? P_ACT_TASKS : 1];
#pragma unroll
    for (int i = 0; i < P_ACT_TASKS; i++) {
        if (!on[i]) continue;
        const uint4* src = reinterpret_cast<const uint4*>(xq + row[i] * cols + b[i] * QK);
        in[i][0] = src[0], in[i][1] = src[1];
        d[i] = xs[row[i] * nbp + b[i]];
        if (Q4) su[Q4 ? i : 0] = xsum[row[i] * nbp + b[i]];
    }
#pragma unroll
    for (int i = 0; i < P_ACT_TASKS; i++) {
        if (!on[i]) continue;
        uint8_t* dst = reinterpret_cast<uint8_t*>(xt + size_t(tile.row0) * cols + size_t(b[i]) * N * 32) + f16_tile_offset(N, n[i], 0);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint4 v = in[i][k / 2];
            const uint2 f0 = f16_from_s8(k & 1 ? v.z : v.x), f1 = f16_from_s8(k & 1 ? v.w : v.y);
            *reinterpret_cast<uint4*>(dst + k * N * 16) = make_uint4(f0.x, f0.y, f1.x, f1.y);
        }
        const size_t so = size_t(tile.row0) * nb + size_t(b[i]) * N + scale_place(n[i]);
        xst[so] = d[i];
        if (Q4) xsumt[so] = su[Q4 ? i : 0];
    }
}

}  // namespace

void init_kernels_prefill() {
    auto opt_in = [](auto kernel, size_t bytes) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
    };
    opt_in(expert_prefill_kernel<false, true>, Stage<false>::SMEM);
    opt_in(expert_prefill_kernel<false, false>, Stage<false>::SMEM);
    opt_in(expert_prefill_kernel<false, false, true>, Stage<false>::SMEM);
    opt_in(expert_prefill_kernel<true, true>, Stage<true>::SMEM);
    opt_in(expert_prefill_kernel<true, false>, Stage<true>::SMEM);
    opt_in(expert_prefill_kernel<true, false, true>, Stage<true>::SMEM);
}

int prefill_row_tiles(const MoeDims& d, bool gate_up) {
    return gate_up ? (d.inter + 63) / 64 : (d.hidden + P_ROWS - 1) / P_ROWS;
}

size_t prefill_weight_bytes(const MoeDims& d, bool gate_up) {
    const int cols = gate_up ? d.hidden : d.inter;
    return size_t(d.experts) * prefill_row_tiles(d, gate_up) * (cols / QK) * P_A_BLOCK;
}

size_t prefill_scale_elems(const MoeDims& d, bool gate_up) {
    const int cols = gate_up ? d.hidden : d.inter;
    return size_t(d.experts) * prefill_row_tiles(d, gate_up) * P_ROWS * (cols / QK);
}

int prefill_tile_columns(const PrefillWeights& w) { return prefill_columns(w.gu_c || w.dn_c); }

// Bounds over every routing: an expert adds at most one tile beyond its whole ones, and pads by up to 63 rows.
int prefill_max_token_tiles(int slots, int experts, bool q4) {
    return slots / prefill_columns(q4) + std::min(slots, experts);
}
size_t prefill_max_rows(int slots, int experts) { return size_t(slots) + 63 * size_t(std::min(slots, experts)); }

void tile_prefill_weights(const MoeDims& d, const MatrixDev& m, bool gate_up, uint16_t* wt, float* wd, float* wc,
                          cudaStream_t stream) {
    const int cols = gate_up ? d.hidden : d.inter;
    const int rpe = gate_up ? 2 * d.inter : d.hidden;
    const int rts = prefill_row_tiles(d, gate_up);
    const dim3 grid(unsigned(d.experts * rts), unsigned((cols / QK + P_WT_BLOCKS - 1) / P_WT_BLOCKS));
    const uint8_t* data = static_cast<const uint8_t*>(m.data);
    if (m.kind == 1) {
        if (gate_up) tile_prefill_weights_kernel<false, true><<<grid, 256, 0, stream>>>(data, m.scales, cols, rpe, rts, wt, wd, wc);
        else tile_prefill_weights_kernel<false, false><<<grid, 256, 0, stream>>>(data, m.scales, cols, rpe, rts, wt, wd, wc);
    } else {
        if (gate_up) tile_prefill_weights_kernel<true, true><<<grid, 256, 0, stream>>>(data, m.scales, cols, rpe, rts, wt, wd, wc);
        else tile_prefill_weights_kernel<true, false><<<grid, 256, 0, stream>>>(data, m.scales, cols, rpe, rts, wt, wd, wc);
    }
}

// One of the two grouped products, gate_up first: it reads the 8-bit rows through
// slot_token and leaves the SwiGLU rows in s.ht / hst / hsumt, as tiles; down reads those.
int launch_prefill(const MoeDims& d, bool gate_up, bool q4, const PrefillWeights& w, const PrefillScratch& s,
                   const Workspace& ws, int slots, float* out, const uint32_t* out_rows, cudaStream_t stream,
                   float* const* peer_out, int peer_ranks, uint32_t peer_rows) {
    const int cols = gate_up ? d.hidden : d.inter;
    const int nb = cols / QK, nbp = (nb + 7) / 8 * 8;
    const bool narrow = w.gu_c || w.dn_c;  // one tile list serves both products
    const int max_tiles = prefill_max_token_tiles(slots, d.experts, narrow);
    int launched = 0;
    if (gate_up) {
        if (!ws.tiles) {
            launch_overlapped(build_token_tiles_kernel, dim3(1), dim3(MAX_EXPERTS), size_t(0), stream,
                              static_cast<const uint32_t*>(ws.counts), static_cast<const uint32_t*>(ws.offsets), d.experts,
                              prefill_columns(narrow), s.tiles, s.tile_count);
            launched++;
        }
        launch_overlapped(q4 ? tile_activations_kernel<true> : tile_activations_kernel<false>,
                          dim3(max_tiles, (nb + P_ACT_BLOCKS - 1) / P_ACT_BLOCKS), dim3(256), size_t(0), stream,
                          static_cast<const int8_t*>(ws.xq), static_cast<const float*>(ws.xs),
                          static_cast<const float*>(ws.xsum), static_cast<const uint32_t*>(ws.slot_token), cols, nbp,
                          static_cast<const TokenTile*>(s.tiles), static_cast<const int*>(s.tile_count), s.xt, s.xst,
                          s.xsumt);
        launched++;
    }
    PrefillArgs a{};
    a.wt = gate_up ? w.gu_t : w.dn_t;
    a.wd = gate_up ? w.gu_d : w.dn_d;
    a.wc = gate_up ? w.gu_c : w.dn_c;
    a.xt = gate_up ? s.xt : s.ht;
    a.xst = gate_up ? s.xst : s.hst;
    a.xsumt = gate_up ? s.xsumt : s.hsumt;
    a.tiles = s.tiles;
    a.tile_count = s.tile_count;
    a.nb = nb;
    a.row_tiles = prefill_row_tiles(d, gate_up);
    a.out_cols = gate_up ? d.inter : d.hidden;
    a.xt_out = s.ht, a.xst_out = s.hst, a.xsumt_out = s.hsumt;
    a.out = out;
    a.out_rows = out_rows;
    a.one = 1.0f;
    a.status = ws.status;
    PrefillPeer pp{};
    const bool to_peers = peer_out && !gate_up;
    if (to_peers) {
        for (int r = 0; r < peer_ranks && r < MAX_PEERS; r++) pp.out[r] = peer_out[r];
        pp.ranks = peer_ranks;
        pp.rows = peer_rows;
    }
    const int sms = ws.sms > 0 ? ws.sms : 148;
    const dim3 grid(unsigned(std::min<long long>(sms, (long long)max_tiles * a.row_tiles))), block(P_THREADS);
    const size_t smem = q4 ? Stage<true>::SMEM : Stage<false>::SMEM;
    if (to_peers)
        launch_overlapped(q4 ? expert_prefill_kernel<true, false, true> : expert_prefill_kernel<false, false, true>, grid, block,
                          smem, stream, a, pp);
    else if (gate_up)
        launch_overlapped(q4 ? expert_prefill_kernel<true, true> : expert_prefill_kernel<false, true>, grid, block, smem,
                          stream, a, NoPeer{});
    else
        launch_overlapped(q4 ? expert_prefill_kernel<true, false> : expert_prefill_kernel<false, false>, grid, block, smem,
                          stream, a, NoPeer{});
    return launched + 1;
}

}  // namespace tc
