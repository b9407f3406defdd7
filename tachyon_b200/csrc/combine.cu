// Weighted combine / unpermute, fused with the residual add.
//
// The CPU path walks experts in ascending index and, for each token routed to
// the expert, does proj[token] += gate * expert_out (src/model.rs:484,
// 513-519; axpy rounds the product before the add, src/kernels.rs:606-610),
// starting from zeros; its caller then adds proj to the residual stream
// (src/model.rs:681). So a token's k contributions are summed in ascending
// expert order, not in the router's score order: each CTA ranks its token's
// picks by expert index and adds them in that order.
//
// Bound by HBM: t k rows of f32 in, t rows read and written. What keeps it from that is a CTA's chain of trips to memory
// (picks, rows, residual row), during two of which nothing large is on its way: so the residual row and all that
// belongs to the picks are asked for together, and a thread takes 16 bytes of the row (256 threads went over a row of 1536
// floats twice, the second time half empty). 4096 tokens of the 1b shape 37 -> 33 us, 2047 of the 3b shape 29.5 -> 25,
// 4096 of 2048 columns 62 -> 60: 167, 126 and 335 MB, 5.0 to 5.6 TB/s.
#include "common.cuh"

namespace tc {

namespace {

constexpr int COMBINE_THREADS = 512;  // at most: 16 bytes of the row a thread

__global__ void __launch_bounds__(COMBINE_THREADS)
combine_kernel(const uint32_t* __restrict__ ids, const float* __restrict__ gates,
               const uint32_t* __restrict__ pos, const float* out, int hidden, int topk,
               float* y, const PeerWait pw) {
    // (`out` without __restrict__: in the peer-memory exchange other GPUs store these rows
    // while this kernel is already resident, up to the wait below.)
    __shared__ uint32_t s_pos[MAX_TOPK];
    __shared__ float s_gate[MAX_TOPK];
    const int token = blockIdx.x, tid = threadIdx.x;
    grid_launch_dependents();
    grid_dependency_wait();
    if (pw.flags) {  // expert outputs arrive from other ranks: all of them have signalled this block
        if (tid < pw.ranks) peer_wait(pw, tid);
        __syncthreads();
    }
    float* yr = y + size_t(token) * hidden;
    float4 y_ahead = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid * 4 < hidden) y_ahead = *reinterpret_cast<const float4*>(yr + tid * 4);
    if (tid < 32) {
        const size_t slot = size_t(token) * topk + min(tid, topk - 1);
        const uint32_t mine = ids[slot], p = pos[slot];
        const float g = gates[slot];
        int rank = 0;
        for (int j = 0; j < topk; j++) rank += __shfl_sync(0xffffffffu, mine, j) < mine ? 1 : 0;
        if (tid < topk) s_pos[rank] = p, s_gate[rank] = g;
    }
    __syncthreads();
    for (int c = tid * 4; c < hidden; c += int(blockDim.x) * 4) {
        float4 proj = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
        for (int j = 0; j < topk; j++) {
            const float g = s_gate[j];
            const float4 v = *reinterpret_cast<const float4*>(out + size_t(s_pos[j]) * hidden + c);
            proj.x = proj.x + g * v.x;
            proj.y = proj.y + g * v.y;
            proj.z = proj.z + g * v.z;
            proj.w = proj.w + g * v.w;
        }
        float4 r = c == tid * 4 ? y_ahead : *reinterpret_cast<float4*>(yr + c);
        r.x = r.x + proj.x;
        r.y = r.y + proj.y;
        r.z = r.z + proj.z;
        r.w = r.w + proj.w;
        *reinterpret_cast<float4*>(yr + c) = r;
    }
}

}  // namespace

int launch_combine(const MoeDims& d, int t, Workspace& ws, float* y, cudaStream_t stream) {
    const int threads = min(COMBINE_THREADS, (d.hidden / 4 + 31) / 32 * 32);
    launch_overlapped(combine_kernel, dim3(t), dim3(threads), size_t(0), stream,
                      static_cast<const uint32_t*>(ws.ids), static_cast<const float*>(ws.gates),
                      static_cast<const uint32_t*>(ws.pos), static_cast<const float*>(ws.out), d.hidden, d.topk, y,
                      ws.combine_wait);
    return 1;
}

}  // namespace tc

