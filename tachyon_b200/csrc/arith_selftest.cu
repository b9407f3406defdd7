// Self-check of the two pieces of arithmetic that stand in for a slower exact form in the kernels' inner parts:
// silu2 (a packed, correctly rounded division) over every float, and div_small (a small integer division on
// the float unit) over every pair a block's partition can ask for. Used by the test-suite through
// tc_arith_selftest; 2^33 and 2^32 evaluations, a fraction of a second together.
#include "experts_common.cuh"

namespace tc {

namespace {

constexpr uint32_t MOST_DIVISOR = 4096;

__device__ __forceinline__ void add_counts(unsigned long long* out, unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

// out[0]: values compared (both halves of the pair), out[1]: those that differ from the IEEE division.
__global__ void __launch_bounds__(256) silu2_check_kernel(float one_value, unsigned long long* out) {
    const float2 one = make_float2(one_value, one_value);
    unsigned long long compared = 0, different = 0;
    const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < (1ull << 32); i += step) {
        const float g = __uint_as_float(uint32_t(i));
        const float want = __fdiv_rn(g, 1.0f + exp_poly(-g));
#pragma unroll
        for (int half = 0; half < 2; half++) {
            bool usable = true;
            const float2 r = silu2(half ? make_float2(1.0f, g) : make_float2(g, 1.0f), one, usable);
            const float got = half ? r.y : r.x;
            if (!usable) continue;  // (the caller divides)
            compared++;
            different += __float_as_uint(got) != __float_as_uint(want) && !(isnan(got) && isnan(want));
        }
    }
    add_counts(out, compared);
    add_counts(out + 1, different);
}

// A CTA per divisor; out: quotients that differ from the integer division.
__global__ void __launch_bounds__(256) div_small_check_kernel(unsigned long long* out) {
    const unsigned b = blockIdx.x + 1;
    unsigned long long different = 0;
    for (unsigned a = threadIdx.x; a < DIV_SMALL; a += blockDim.x) different += div_small(a, b) != a / b;
    add_counts(out, different);
}

}  // namespace

// out (device, zeroed): silu2 values compared, silu2 values that differ, div_small quotients that differ.
int launch_arith_selftest(int sms, unsigned long long* out, cudaStream_t stream) {
    silu2_check_kernel<<<sms * 8, 256, 0, stream>>>(1.0f, out);
    div_small_check_kernel<<<MOST_DIVISOR, 256, 0, stream>>>(out + 2);
    return 2;
}

}  // namespace tc
