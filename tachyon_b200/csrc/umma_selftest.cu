// Self-check of the tcgen05 building blocks as the grouped kernels use them: one block of 32
// columns of 8-bit values held as f16, 128 x N, as two K = 16 products from shared memory
// into tensor memory, read back to global memory. Used by the test-suite (through
// tc_umma_selftest) to pin the descriptor encodings, the tile layout and the exactness of the
// sums that those kernels rely on. Every wait is bounded.
#include "experts_common.cuh"
#include "umma.cuh"

namespace tc {

namespace {

template <int N>
__global__ void __launch_bounds__(128, 1)
umma_selftest_kernel(const uint16_t* __restrict__ a_tile, const uint16_t* __restrict__ b_tile, float* __restrict__ d_out,
                  int* __restrict__ status) {
    __shared__ __align__(128) uint8_t s_a[128 * 64];
    __shared__ __align__(128) uint8_t s_b[N * 64];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // Tiles are already in the canonical order in global memory: plain copy.
    for (int i = tid; i < 128 * 64 / 16; i += 128)
        reinterpret_cast<uint4*>(s_a)[i] = reinterpret_cast<const uint4*>(a_tile)[i];
    for (int i = tid; i < N * 64 / 16; i += 128)
        reinterpret_cast<uint4*>(s_b)[i] = reinterpret_cast<const uint4*>(b_tile)[i];
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Generic-proxy writes above must be visible to the tensor core's async-proxy reads.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        umma::tmem_alloc(&s_tmem, 64 < N ? 128 : 64);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem;
    if (warp == 0) {  // an elected lane of a converged warp, as the issuing warp of those kernels
        const uint32_t da = umma::smem_desc_low(smem_addr(s_a), 128 * 16), db = umma::smem_desc_low(smem_addr(s_b), N * 16);
        if (umma::elect_one()) {
#pragma unroll
            for (int h = 0; h < 2; h++)
                umma::mma_f16_low(tmem, da + h * 128 * 2, db + h * N * 2, umma::idesc_f16(128, N), uint32_t(h));
            umma::commit(&s_bar);
        }
        __syncwarp();
    }
    const bool landed = mbar_wait_bounded(&s_bar, 0);
    umma::fence_after_sync();
    if (landed) {
        // A half of the rows at a time, in the two widths those kernels use: 32 columns, and twice 16, of every 64.
        const uint32_t base = tmem + (uint32_t(warp * 32) << 16);
        auto read = [&](int c0, int h, auto& v) {
            constexpr int n = sizeof(v) / sizeof(float);
            umma::ld_half_f32(base + (uint32_t(h) << 20) + c0, v);
            umma::wait_ld(v);
#pragma unroll
            for (int j = 0; j < n / 4; j++)
#pragma unroll
                for (int r = 0; r < 2; r++)
                    *reinterpret_cast<float2*>(d_out + (warp * 32 + h * 16 + r * 8 + (lane >> 2)) * N + c0 + 8 * j + 2 * (lane & 3)) =
                        make_float2(v[4 * j + 2 * r], v[4 * j + 2 * r + 1]);
        };
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 64) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float v[16], lo[8], hi[8];
                read(c0, h, v);
                read(c0 + 32, h, lo);
                read(c0 + 48, h, hi);
            }
        }
    } else if (tid == 0) {
        atomicExch(status, ERR_COPY_WAIT_TIMEOUT);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 64 < N ? 128 : 64);
}

}  // namespace

// a_tile: 128 x 32 f16, b_tile: n x 32 f16, both in the canonical tile order (umma::f16_tile_offset);
// d_out: 128 x n floats row-major. n is 64 or 128.
int launch_umma_selftest(const uint16_t* a_tile, const uint16_t* b_tile, int n, float* d_out, int* status,
                      cudaStream_t stream) {
    if (n == 64)
        umma_selftest_kernel<64><<<1, 128, 0, stream>>>(a_tile, b_tile, d_out, status);
    else if (n == 128)
        umma_selftest_kernel<128><<<1, 128, 0, stream>>>(a_tile, b_tile, d_out, status);
    else
        return -1;
    return 1;
}

}  // namespace tc
