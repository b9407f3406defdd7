"""The edges of the kernels' tiles and of the rules that choose a variant: one token more or less than a tile, an
odd number of 32-value blocks per row, router matrices that fit on chip or not, more experts than a warp ranks at
once, experts without a token; a call over host buffers on both sides of its rule. Against the oracle."""
import numpy as np
import pytest

from tachyon_b200 import synth, weights, workloads
from tachyon_b200.workloads import MoeShape
from test_gpu_parity import check_block, ctx, layer_weights, make_layer, oracle_moe  # noqa: F401

pytestmark = pytest.mark.gpu

ODD_Q8 = MoeShape("odd-q8", 288, 8, 2, 160, fmt="q8")        # 9 and 5 blocks per row; rows end inside a tile of 128
ODD_Q4 = MoeShape("odd-q4", 288, 8, 2, 160, fmt="q4")
ONE_BLOCK = MoeShape("one-block", 32, 3, 1, 32, fmt="q8")    # one block per row, one pick
ODD_EXPERTS = MoeShape("experts-37", 96, 37, 5, 32, fmt="q8")
PAST_64 = MoeShape("experts-65", 64, 65, 8, 32, fmt="q8")    # one expert more than two per lane
MANY_PICKS = MoeShape("picks-31", 96, 31, 31, 32, fmt="q8")  # every expert by every token: 496 runs of 8 at 128 tokens
WIDE = MoeShape("wide-router", 2048, 64, 8, 32, fmt="q4")    # 256 KB of router matrix: staged in parts


@pytest.mark.parametrize("shape,t,skewed", [
    # One kernel per block: a token, an odd few, and both sides of 32 tokens and of the largest batch.
    (ODD_Q4, 1, False), (ODD_EXPERTS, 3, False), (PAST_64, 31, True), (ONE_BLOCK, 33, False), (WIDE, 127, True),
    (ODD_Q8, 129, False), (MANY_PICKS, 128, False), (MANY_PICKS, 90, True),
    # Tensor-core tiles: whole ones, one token past them, experts with hardly any.
    (ODD_Q8, 256, False), (ODD_Q4, 257, False), (ODD_Q8, 1025, True), (ODD_Q4, 770, True), (ONE_BLOCK, 193, False),
    # Both sides of the switch to the tensor cores past 128 tokens.
    (PAST_64, 129, True), (WIDE, 129, True),
    # Router tiles of 4 and 8 tokens, each with a remainder; the dispatch past one CTA's batch.
    (ODD_EXPERTS, 257, False), (ODD_EXPERTS, 595, False), (ODD_EXPERTS, 1187, True), (PAST_64, 1191, True),
    (WIDE, 259, False), (WIDE, 597, True), (WIDE, 1189, False), (ONE_BLOCK, 2049, False),
], ids=lambda v: v.name if isinstance(v, MoeShape) else str(v))
def test_blocks_at_the_edges(oracle, ctx, shape, t, skewed):
    lw = layer_weights(oracle, shape, 17)
    bias = synth.zipf_router_bias(17, shape.experts) if skewed else None
    check_block(oracle, ctx, shape, lw, workloads.hidden_states(shape, t, seed=t), bias=bias, arith="fast")


def block_in_one_and_by_100(ctx, layer, x, norm):
    """Everything a block leaves behind, of the whole batch (the router's tiles) and of 100 tokens at a time (the router of
    one token), both on the kernels that read the router's 8-bit rows with their padded scales."""
    def run(rows):
        y = ctx.to_device(rows)
        layer.block(norm, 1e-6, y)
        ids, gates, _, logits = layer.last_routing(len(rows))
        out = [ids, gates, logits, y.get()]
        y.free()
        return out

    ctx.set_decode_block(False)
    ctx.set_prefill_threshold(1 << 30)
    try:
        whole = run(x)
        dispatch = layer.last_dispatch(len(x))
        parts = [run(x[lo:lo + 100]) for lo in range(0, len(x), 100)]
    finally:
        ctx.set_decode_block(True)
        ctx.set_prefill_threshold(16)
    return whole, [np.concatenate(p) for p in zip(*parts)], dispatch


@pytest.mark.parametrize("hidden,experts,topk,fmt", [
    (96, 31, 5, "q4"), (160, 40, 8, "q8"), (544, 64, 8, "q4"), (96, 65, 9, "q4"), (1056, 130, 8, "q8"), (64, 256, 32, "q8"),
])
@pytest.mark.parametrize("t", [131, 261, 500, 803, 1601, 3200])
def test_router_tiles_match_the_router_of_one_token(oracle, ctx, hidden, experts, topk, fmt, t):
    """Every tile size with a remainder, experts in one CTA and split over two to four, rows that end inside a chunk and inside
    a super-block, and experts of equal rows (so equal logits): the block of the same tokens 100 at a time, bit for bit,
    and their order by expert."""
    router = synth.normal(41, synth.STREAM_ROUTER, experts * hidden).reshape(experts, hidden) * 0.1
    router[experts // 2] = router[3]
    router[experts - 1] = router[0]
    shape = MoeShape("tiles", hidden, experts, topk, 32, fmt=fmt)
    lw = layer_weights(oracle, shape, 3)
    lw = workloads.LayerWeights(weights.Matrix.from_f32(router.reshape(-1), experts, hidden, "bf16"), lw.gate_up, lw.down)
    x = workloads.hidden_states(shape, t, seed=t)
    x[5] = 0.0  # (all logits equal)
    norm = ctx.to_device((1.0 + 0.1 * synth.normal(7, synth.STREAM_HIDDEN, hidden)).astype(np.float32))
    ctx.set_arithmetic(ctx.ARITH_FAST)
    # Longer rows before: what they leave in the scratch must not show.
    long = MoeShape("long", 2080, 2, 1, 32, fmt=fmt)
    before = make_layer(ctx, layer_weights(oracle, long, 3), 1, t)
    layer = make_layer(ctx, lw, topk, t)
    try:
        rows = ctx.to_device(workloads.hidden_states(long, t, seed=1))
        before.block(ctx.to_device(np.ones(2080, np.float32)), 1e-6, rows)
        rows.free()
        whole, parts, (offsets, perm) = block_in_one_and_by_100(ctx, layer, x, norm)
        picks = whole[0].reshape(-1)
        assert np.array_equal(perm, np.argsort(picks, kind="stable"))
        assert np.array_equal(offsets[1:], np.cumsum(np.bincount(picks, minlength=experts)))
        for a, b in zip(whole, parts):
            assert np.array_equal(a, b)
    finally:
        layer.free()
        before.free()


@pytest.mark.parametrize("experts", [32, 130])
@pytest.mark.parametrize("t", [131, 1601, 4000])
def test_router_tiles_on_rows_that_are_not_finite(oracle, ctx, experts, t):
    """NaN, infinite, tiny and overflowing rows: the same picks, gates and output rows as from the router of one token,
    and the rows beside them untouched by it."""
    shape = MoeShape("odd-rows", 160, experts, 4, 32, fmt="q8")
    lw = layer_weights(oracle, shape, 3)
    clean = workloads.hidden_states(shape, t, seed=t)
    x = clean.copy()
    odd = [3, 17, 40, 66, 90, 127, t - 1]
    x[3, 7] = np.nan
    x[17, ::3] = np.inf
    x[40, 5] = -np.inf
    x[66] = 1e-41
    x[90] = 3e38
    x[127] = -0.0
    x[t - 1] = np.nan
    norm = ctx.to_device((1.0 + 0.1 * synth.normal(7, synth.STREAM_HIDDEN, 160)).astype(np.float32))
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, 4, t)
    try:
        whole, parts, _ = block_in_one_and_by_100(ctx, layer, x, norm)
        for a, b in zip(whole, parts):
            assert np.array_equal(a, b, equal_nan=True)
        assert all(len(set(p)) == 4 and max(p) < experts for p in whole[0].tolist())
        rest = np.setdiff1d(np.arange(t), odd)
        for a, b in zip(whole, block_in_one_and_by_100(ctx, layer, clean, norm)[0]):
            assert np.array_equal(a[rest], b[rest])
    finally:
        layer.free()


@pytest.mark.parametrize("t", [1, 33, 128, 129, 257, 800, 1600, 3200])
def test_the_norms_weight_may_stand_at_any_float(oracle, ctx, t):
    """A norm's weight that is a slice of a packed buffer, 4, 8 or 12 bytes past a 16-byte boundary: the same bits as
    from an aligned one in every kernel that reads it (the one-kernel block, the router of a token, all router tiles)."""
    shape = MoeShape("slice", 544, 8, 2, 32, fmt="q8")
    lw = layer_weights(oracle, shape, 17)
    x = workloads.hidden_states(shape, t, seed=t)
    norm = (1.0 + 0.1 * synth.normal(7, synth.STREAM_HIDDEN, shape.hidden)).astype(np.float32)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, shape.topk, t)

    def block(off):
        packed = ctx.to_device(np.concatenate([np.full(off, 7.0, np.float32), norm, np.full(4, 7.0, np.float32)]))
        assert packed.ptr % 16 == 0
        y = ctx.to_device(x)
        assert ctx.lib.tc_moe_block(layer.handle, packed.ptr + 4 * off, 1e-6, t, y.ptr) == 0
        out = (y.get(), *layer.last_routing(t))
        for d in (y, packed):
            d.free()
        return out

    try:
        for one_kernel in (True, False):
            ctx.set_decode_block(one_kernel)
            aligned = block(0)
            for off in (1, 2, 3):
                for a, b in zip(aligned, block(off)):
                    assert np.array_equal(a, b)
    finally:
        ctx.set_decode_block(True)
        layer.free()


@pytest.mark.parametrize("experts,topk,t", [
    (3, 1, 8192), (3, 1, 8193), (3, 2, 8192), (3, 2, 17000), (200, 2, 8192), (200, 2, 8193), (200, 1, 20001),
])
def test_dispatch_of_an_expert_with_more_slots_than_are_held(oracle, ctx, experts, topk, t):
    """An expert's slots go through shared memory up to 8192 of them and straight to their places beyond: every token on
    expert 1, so as many slots, one more, and twice as many, beside the rest of the slots."""
    shape = MoeShape("crowd", 32, experts, topk, 32, fmt="q8")
    lw = layer_weights(oracle, shape, 3)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, topk, t)
    layer.set_router_bias(np.where(np.arange(experts) == 1, 1e6, 0.0).astype(np.float32))
    x = ctx.to_device(workloads.hidden_states(shape, t, seed=t))
    y = ctx.to_device(np.zeros((t, 32), np.float32))
    try:
        layer.forward(x, y)
        ids = layer.last_routing(t)[0]
        offsets, perm = layer.last_dispatch(t)
        assert np.array_equal(ids[:, 0], np.full(t, 1))
        assert np.array_equal(perm, np.argsort(ids.reshape(-1), kind="stable"))
        assert np.array_equal(offsets[1:], np.cumsum(np.bincount(ids.reshape(-1), minlength=experts)))
    finally:
        layer.free()
        x.free()
        y.free()


@pytest.mark.parametrize("t", [1, 128, 129])
def test_host_buffers_at_the_edges(oracle, ctx, t):
    lw = layer_weights(oracle, ODD_Q8, 17)
    x = workloads.hidden_states(ODD_Q8, t, seed=t)
    y = np.ones_like(x)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, ODD_Q8.topk, t)
    try:
        layer.forward_host(x, y)
    finally:
        layer.free()
    want = 1.0 + oracle_moe(oracle, lw, x, ODD_Q8.topk).proj
    assert np.abs(y - want).max() <= 2e-3


def test_copies_take_device_and_page_locked_memory_only(ctx):
    """Pageable memory is refused either way round, also inside a capture, which stays usable."""
    from tachyon_b200 import cuda

    n = 1024
    host, plain = ctx.host_empty(n), np.full(n, 7.0, np.float32)
    a, b = ctx.to_device(np.arange(n, dtype=np.float32)), ctx.to_device(np.zeros(n, np.float32))

    def refused(dst, src):
        with pytest.raises(cuda.TachyonCudaError, match="page-locked"):
            ctx.copy_bytes(dst, src, 4 * n)

    refused(a.ptr, plain.ctypes.data)
    refused(plain.ctypes.data, a.ptr)
    ctx.capture_begin()
    refused(a.ptr, plain.ctypes.data)
    refused(plain.ctypes.data, a.ptr)
    ctx.copy_bytes(b.ptr + 4, a.ptr + 4, 4 * n - 4)
    ctx.copy_bytes(host.ptr, b.ptr, 4 * n)
    g = ctx.capture_end()
    g.launch()
    ctx.sync()
    assert np.array_equal(a.get(), np.arange(n)) and np.array_equal(host.array, np.arange(n)) and np.all(plain == 7.0)
    g.free()
    for d in (host, a, b):
        d.free()


def test_more_short_runs_than_the_kernel_lists(oracle, ctx):
    """The run-walking form where runs of 8 tokens look cheapest and there would be 336 of them, 16 more than its tables
    once held: the runs past the end were left out. The router is the identity, so a row's largest elements
    are its picks and every expert gets the tokens asked for."""
    counts = [1] * 230 + [30] * 25 + [44]
    shape = MoeShape("runs", 256, len(counts), 8, 32, fmt="q8")
    t = sum(counts) // shape.topk
    lw = layer_weights(oracle, shape, 17)
    lw = workloads.LayerWeights(weights.Matrix.from_f32(np.eye(256, dtype=np.float32).ravel(), 256, 256, "bf16"), lw.gate_up, lw.down)
    x = 0.1 * workloads.hidden_states(shape, t, seed=3)
    x[np.arange(sum(counts)) % t, np.repeat(np.arange(len(counts)), counts)] += 4.0
    check_block(oracle, ctx, shape, lw, x, arith="fast")


@pytest.mark.parametrize("t", [20, 100, 300])
def test_a_layer_that_cannot_be_had_leaves_the_others_working(oracle, ctx, t):
    """Scratch is shared by a context's layers and grows with them. A layer whose scratch is more than the device has
    is refused; the layers that are there, and graphs captured on them, go on as before."""
    from tachyon_b200 import cuda

    many = MoeShape("many", 32, 256, 1, 32, fmt="q8")
    lw, other = layer_weights(oracle, ODD_Q8, 17), layer_weights(oracle, many, 17)
    x = workloads.hidden_states(ODD_Q8, t, seed=t)
    ctx.set_arithmetic(ctx.ARITH_FAST)
    layer = make_layer(ctx, lw, ODD_Q8.topk, t)
    xd, yd = ctx.to_device(x), ctx.to_device(np.zeros_like(x))
    ctx.capture_begin()
    layer.forward(xd, yd)
    g = ctx.capture_end()
    with pytest.raises(cuda.TachyonCudaError, match="memory"):
        make_layer(ctx, other, many.topk, 1 << 28)  # 256 GB of logits
    g.launch()
    ctx.sync()
    first = yd.get()
    yd.set(np.zeros_like(x))
    layer.forward(xd, yd)
    ctx.sync()
    assert np.array_equal(yd.get(), first)
    assert np.abs(first - oracle_moe(oracle, lw, x, ODD_Q8.topk).proj).max() <= 2e-3
    g.free()
    layer.free()
