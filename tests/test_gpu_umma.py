"""The tcgen05 (tensor memory) building blocks as the expert kernels use them: a block of 8-bit values, as f16, must
give the exact integer product. And the arithmetic that stands in for exact divisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128])
def test_one_tcgen05_block_is_exact(n):
    from tachyon_b200 import build, cuda

    build.build()
    ctx = cuda.Context(0)
    rng = np.random.default_rng(n)
    a = rng.integers(-127, 128, size=(128, 32), dtype=np.int8)
    b = rng.integers(-127, 128, size=(n, 32), dtype=np.int8)
    a[:2], b[:2] = -128, -128  # (the largest sums: 32 * 2^14)
    got = ctx.umma_selftest(a, b)
    want = a.astype(np.int32) @ b.astype(np.int32).T
    assert want.max() == 1 << 19
    assert np.array_equal(got, want)
    ctx.close()


def test_packed_and_float_unit_divisions_are_exact():
    """The packed SwiGLU division has the IEEE division's bits for every float it is used for (1e-18 to 1e18 in
    magnitude, not below -41: 1.55e9 floats and the NaNs, in either half of a pair), and the partition's division
    is the integer one."""
    from tachyon_b200 import build, cuda

    build.build()
    ctx = cuda.Context(0)
    n = ctx.arith_selftest()
    assert n["silu_compared"] > 2 * 1_500_000_000
    assert n["silu_different"] == 0
    assert n["quotients_different"] == 0
    ctx.close()
