"""The tcgen05 (tensor memory) expert kernels against the oracle and against the
bandwidth-oriented kernels: same fma chain per output, so the same bits.

Past the one-kernel block's 128 tokens the library picks the tensor-core kernels from an
average of 16 tokens per expert; the tests force either path with the threshold, and
below 129 tokens with the one-kernel block off."""
import numpy as np
import pytest

from tachyon_b200 import synth, workloads
from tachyon_b200.workloads import MoeShape
from test_gpu_parity import check_block, ctx, layer_weights, make_layer  # noqa: F401

pytestmark = pytest.mark.gpu

NEVER, DEFAULT = 1 << 30, 16


def forward(ctx, layer, x, y0):
    xd, yd = ctx.to_device(x), ctx.to_device(y0)
    layer.forward(xd, yd)
    ctx.sync()
    y = yd.get()
    xd.free()
    yd.free()
    return y


@pytest.fixture
def always_prefill(ctx):
    ctx.set_prefill_threshold(0)
    yield ctx
    ctx.set_prefill_threshold(DEFAULT)


@pytest.mark.parametrize("shape,t", [
    (MoeShape("small-q8", 256, 8, 2, 96, fmt="q8"), 300),    # ragged row tile (96 rows of 128), one chunk
    (MoeShape("small-q4", 512, 16, 4, 192, fmt="q4"), 333),  # 4-bit offsets, ragged token tiles
    (MoeShape("1b-q8", 1024, 32, 8, 512, fmt="q8"), 512),    # operand ring and TMEM ring wrap
    (MoeShape("3b-q4", 1536, 40, 8, 512, fmt="q4"), 200),
])
def test_prefill_kernels_meet_the_oracle_bars(oracle, always_prefill, shape, t):
    lw = layer_weights(oracle, shape, 11)
    x = workloads.hidden_states(shape, t, seed=11)
    check_block(oracle, always_prefill, shape, lw, x, arith="fast")


@pytest.mark.parametrize("fmt", ["q8", "q4"])
def test_both_kernel_families_give_the_same_bits(oracle, ctx, fmt):
    """Also with a skewed router: experts with no token, one token, several 64-token tiles."""
    shape = MoeShape("skew-small", 256, 64, 8, 64, fmt=fmt)
    lw = layer_weights(oracle, shape, 5)
    bias = synth.zipf_router_bias(5, 64)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    for t in [1, 7, 64, 65, 700, 2048]:
        x = workloads.hidden_states(shape, t, seed=5)
        y0 = synth.normal(9, synth.STREAM_HIDDEN, x.size, layer=1).reshape(x.shape)
        layer = make_layer(ctx, lw, shape.topk, t)
        layer.set_router_bias(bias)
        try:
            default = forward(ctx, layer, x, y0)  # up to 128 tokens: the one-kernel block
            ctx.set_decode_block(False)
            ctx.set_prefill_threshold(NEVER)
            a = forward(ctx, layer, x, y0)
            ctx.set_prefill_threshold(0)
            before = ctx.launch_count()
            b = forward(ctx, layer, x, y0)
            assert ctx.launch_count() - before >= 5  # (the tensor-core kernels tile the activations first)
            b2 = forward(ctx, layer, x, y0)
        finally:
            ctx.set_decode_block(True)
            ctx.set_prefill_threshold(DEFAULT)
            layer.free()
        assert np.array_equal(a, default)
        assert np.array_equal(a, b)
        assert np.array_equal(b, b2)


@pytest.mark.parametrize("fmt", ["q8", "q4"])
@pytest.mark.parametrize("hidden,inter", [(32, 64), (64, 160), (96, 32), (160, 96), (192, 288), (224, 256)])
def test_any_number_of_blocks_gives_the_same_bits(oracle, ctx, fmt, hidden, inter):
    """Rows of 1 to 9 blocks: whole passes of the float loop (four blocks), what is left after them, and chunks of
    one block; token tiles of every width, some not full."""
    shape = MoeShape("blocks", hidden, 6, 2, inter, fmt=fmt)
    lw = layer_weights(oracle, shape, 7)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, shape.topk, 500)
    layer.set_router_bias(synth.zipf_router_bias(7, 6))
    try:
        for t in [33, 130, 500]:
            x = workloads.hidden_states(shape, t, seed=t)
            y0 = np.zeros_like(x)
            ctx.set_decode_block(False)
            ctx.set_prefill_threshold(NEVER)
            a = forward(ctx, layer, x, y0)
            ctx.set_prefill_threshold(0)
            b = forward(ctx, layer, x, y0)
            assert np.array_equal(a, b)
    finally:
        ctx.set_decode_block(True)
        ctx.set_prefill_threshold(DEFAULT)
        layer.free()


def test_default_threshold_switches_by_batch_size(oracle, ctx):
    """Crossing the threshold, or the end of the one-kernel block, must not change a token's output."""
    shape = MoeShape("small-q8", 256, 8, 2, 96, fmt="q8")
    lw = layer_weights(oracle, shape, 11)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    ctx.set_prefill_threshold(DEFAULT)
    x = workloads.hidden_states(shape, 256, seed=3)
    y0 = np.zeros_like(x)
    layer = make_layer(ctx, lw, shape.topk, 256)

    def run(t, launches):
        before = ctx.launch_count()
        y = forward(ctx, layer, x[:t], y0[:t])
        assert ctx.launch_count() - before == launches
        return y

    try:
        big = run(256, 5)      # 64 per expert: tensor-core path
        one = run(40, 1)       # the one-kernel block
        ctx.set_decode_block(False)
        at = run(64, 5)        # 16 per expert: tensor-core path
        below = run(63, 4)     # bandwidth path
    finally:
        ctx.set_decode_block(True)
        layer.free()
    for y in (one, at, below):
        assert np.array_equal(big[:len(y)], y)


def test_scratch_shared_by_layers_only_grows(oracle, ctx):
    """Two layers in one context share the token-tile scratch of the tensor-core path. A
    wide layer is created first, then a narrow one that needs more tiles but fewer bytes
    per tile; the wide layer's next prefill-size block must still fit (and be right)."""
    wide = MoeShape("wide", 1024, 8, 2, 256, fmt="q8")
    narrow = MoeShape("narrow", 256, 16, 4, 64, fmt="q8")
    lw_w, lw_n = layer_weights(oracle, wide, 21), layer_weights(oracle, narrow, 22)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    la = make_layer(ctx, lw_w, wide.topk, 600)
    lb = make_layer(ctx, lw_n, narrow.topk, 1200)
    ctx.set_prefill_threshold(0)
    try:
        for layer, shape, lw, t in [(la, wide, lw_w, 600), (lb, narrow, lw_n, 1200), (la, wide, lw_w, 600)]:
            x = workloads.hidden_states(shape, t, seed=23)
            y0 = np.zeros_like(x)
            got = forward(ctx, layer, x, y0)
            with oracle.fast_arithmetic_model():
                from test_gpu_parity import oracle_moe

                want = oracle_moe(oracle, lw, x, shape.topk).proj
            assert np.abs(got - want).max() <= 2e-3
            assert np.mean(np.all(got == want, axis=1)) > 0.5
    finally:
        ctx.set_prefill_threshold(DEFAULT)
        la.free()
        lb.free()


@pytest.mark.parametrize("fmt", ["q8", "q4"])
def test_decode_only_layers_hold_no_tensor_core_copy(oracle, ctx, fmt):
    """A layer whose every block runs as one kernel does without the tensor-core kernels' copy of its experts
    (2.125 bytes per 8-bit weight, 2.25 with 4-bit offsets). Once a switch makes those kernels reachable the
    copy is there and they run; a layer whose uploaded matrices are gone runs on the bandwidth-oriented
    kernels instead. The same bits every time."""
    import torch

    shape = MoeShape("1b", 1024, 32, 8, 512, fmt=fmt)
    copy = shape.experts * 3 * shape.inter * shape.hidden * (2.125 if fmt == "q8" else 2.25)
    pages = 16 << 20  # (allocations take whole pages of 2 MB)
    lw = layer_weights(oracle, shape, 0)
    x = workloads.hidden_states(shape, 128, seed=31)
    y0 = np.zeros_like(x)
    ctx.set_arithmetic(ctx.ARITH_FAST)

    def launches_of(layer):
        before = ctx.launch_count()
        return forward(ctx, layer, x, y0), ctx.launch_count() - before

    layers = [make_layer(ctx, lw, shape.topk, 129)]  # (the context's scratch has its size from here on)
    try:
        free = [torch.cuda.mem_get_info(ctx.device)[0]]
        for most in (128, 129):  # 129 tokens: one past the one-kernel block
            layers.append(make_layer(ctx, lw, shape.topk, most))
            free.append(torch.cuda.mem_get_info(ctx.device)[0])
        small, large = free[0] - free[1], free[1] - free[2]
        assert abs(large - small - copy) < pages
        one, n = launches_of(layers[1])
        assert n == 1
        detached = make_layer(ctx, lw, shape.topk, 128)
        layers.append(detached)
        detached.detach_experts()
        before = torch.cuda.mem_get_info(ctx.device)[0]
        ctx.set_decode_block(False)  # 32 tokens per expert: the tensor-core kernels, for the layers that can have the copy
        assert abs(before - torch.cuda.mem_get_info(ctx.device)[0] - copy) < pages
        layers.append(make_layer(ctx, lw, shape.topk, 128))
        for layer, kernels in [(layers[1], 5), (layers[2], 5), (detached, 4), (layers[4], 5)]:
            y, n = launches_of(layer)
            assert n == kernels
            assert np.array_equal(y, one)
    finally:
        ctx.set_decode_block(True)
        for layer in layers:
            layer.free()
