"""What a user of this backend has it do, as measurable cases: the MoE blocks of a
Granite model over decode steps and prompt chunks, through the entry points that
Tachyon's forward pass binds (``tachyon_b200.cuda`` over ``include/tachyon_cuda.h``).

A case is a shape (hidden, experts, topk, inter), a weight format, a number of
tokens, a number of layers and the way the blocks are called:

  graph    the layers' blocks on a device-resident residual stream, one captured graph
           per step: how a decode loop runs (``tc_moe_block`` + ``tc_capture_*``)
  serve    ``GraphBuckets.step``: a scheduler's step, rows in from and out to the host,
           the batch padded to its bucket's graph
  host     ``MoeLayer.forward_host``: one block over host buffers, as a host engine
           with a single block off-loaded calls it
  block    the layers' blocks enqueued one by one: a prompt chunk, whose length is new
           each time, so nothing is captured

The shapes are those of ``tachyon_b200/workloads.py``.
"""
import math

import numpy as np
import torch

from tachyon_b200 import cuda, synth
from tachyon_b200.buckets import GraphBuckets

EPS = 1e-6

SHAPES = {
    "1b": {"hidden": 1024, "experts": 32, "topk": 8, "inter": 512},    # granite-1b-a400m
    "3b": {"hidden": 1536, "experts": 40, "topk": 8, "inter": 512},    # granite-3b-a800m
    "skew": {"hidden": 2048, "experts": 64, "topk": 8, "inter": 1024}, # the routing-skew shape
}


def _case(shape, fmt, tokens, layers, call, skewed=False, name=None):
    c = dict(SHAPES[shape], fmt=fmt, tokens=tokens, layers=layers, call=call, skewed=skewed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One sequence generating: the latency of a step.
        _case("1b", "q8", 1, 4, "graph", name="decode-1b-q8-1"),
        # A few sequences: only some of the experts are picked.
        _case("1b", "q8", 8, 4, "graph", name="decode-1b-q8-8"),
        # The headline batch of bench.py.
        _case("1b", "q8", 32, 4, "graph", name="decode-1b-q8-32"),
        # The larger model in 4 bits, as it is shipped to save memory.
        _case("3b", "q4", 16, 4, "graph", name="decode-3b-q4-16"),
        # Busy servers: more sequences than one pass over an expert's tokens takes.
        _case("1b", "q8", 64, 4, "graph", name="decode-1b-q8-64"),
        _case("3b", "q8", 100, 4, "graph", name="decode-3b-q8-100"),
        # A scheduler's step with an odd number of sequences.
        _case("1b", "q8", 13, 4, "serve", name="serve-1b-q8-13"),
        # One block called over host buffers.
        _case("1b", "q8", 4, 1, "host", name="host-1b-q8-4"),
        # Prompt chunks: a short ragged one, a full one (4 x 1024 tokens), a ragged one in 4 bits.
        _case("1b", "q8", 333, 1, "block", name="prefill-1b-q8-333"),
        _case("1b", "q8", 4096, 1, "block", name="prefill-1b-q8-4096"),
        _case("3b", "q4", 2047, 1, "block", name="prefill-3b-q4-2047"),
        # The wide shape with a router that prefers a few experts (Zipf 1.2).
        _case("skew", "q8", 4096, 1, "block", skewed=True, name="prefill-skew-q8-4096"),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    call = rng.choice(["graph"] * 4 + ["block"] * 4 + ["serve", "host"])
    shape = rng.choice(["1b", "1b", "3b", "3b", "skew"])
    fmt = rng.choice(["q8", "q8", "q4"])
    skewed = rng.random() < 0.25
    if call == "block":
        # (As many tokens as keep the work within the largest listed case.)
        tokens = _log_uniform(rng, 129, 4096 if shape == "skew" else 8192)
        return _case(shape, fmt, tokens, 1, call, skewed)
    tokens = _log_uniform(rng, 1, 128)
    layers = 1 if call == "host" or shape == "skew" else rng.choice([2, 3, 4])
    return _case(shape, fmt, tokens, layers, call, skewed)


_context = None


def _ctx():
    """One context per process, as a program has: it owns the stream and the scratch."""
    global _context
    if _context is None:
        _context = cuda.Context(torch.cuda.current_device())
    return _context


class _View:
    """A DeviceArray as torch sees it (no copy)."""

    def __init__(self, array):
        self.array = array
        self.__cuda_array_interface__ = {"shape": array.shape, "typestr": array.dtype.str, "data": (array.ptr, False),
                                         "version": 3}


def _normal_host(gen, n, scale):
    """n draws of N(0, scale^2), made on the GPU, in page-locked host memory."""
    host = torch.empty(n, dtype=torch.float32, pin_memory=True)
    host.copy_(torch.randn(n, generator=gen, device="cuda", dtype=torch.float32).mul_(scale))
    return host.numpy()


def _layer(ctx, case, gen, seed, tokens):
    h, e, i = case["hidden"], case["experts"], case["inter"]
    q = cuda.DeviceMatrix.quantize
    layer = cuda.MoeLayer(ctx, q(ctx, _normal_host(gen, e * h, 0.02), e, h, "bf16"),
                          q(ctx, _normal_host(gen, e * 2 * i * h, 0.02), e * 2 * i, h, case["fmt"]),
                          q(ctx, _normal_host(gen, e * h * i, 0.02), e * h, i, case["fmt"]), case["topk"], tokens)
    if case["skewed"]:
        layer.set_router_bias(synth.zipf_router_bias(seed, e))
    return layer


class _State:
    pass


def prepare(case, seed):
    ctx = _ctx()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t, h, call = case["tokens"], case["hidden"], case["call"]
    s = _State()
    s.ctx, s.call, s.t = ctx, call, t
    most = max(128, t) if call == "serve" else t
    s.layers = [_layer(ctx, case, gen, seed + l, most) for l in range(case["layers"])]
    x = torch.randn(t, h, generator=gen, device="cuda", dtype=torch.float32)
    norms = [(1.0 + 0.1 * torch.randn(h, generator=gen, device="cuda")).cpu().numpy() for _ in s.layers]
    if call == "host":
        s.x = x.cpu().numpy()
        s.y = np.zeros_like(s.x)
        return s
    s.norms = [ctx.to_device(w) for w in norms]
    if call == "serve":
        s.x = x.cpu().numpy()
        s.buckets = GraphBuckets(ctx, s.layers, s.norms, EPS, h)
        s.buckets.graph(s.buckets.bucket_for(t))
        return s
    s.x_in = ctx.to_device(x.cpu().numpy())
    s.x = ctx.empty((t, h))
    s.out = torch.as_tensor(_View(s.x), device="cuda")
    if call == "graph":
        _enqueue(s)
        ctx.sync()
        ctx.capture_begin()
        _enqueue(s)
        s.graph = ctx.capture_end()
    ctx.sync()
    return s


def _enqueue(s):
    s.ctx.copy(s.x, s.x_in)  # the step's hidden states arrive
    for layer, w in zip(s.layers, s.norms):
        layer.block(w, EPS, s.x, t=s.t)  # x += moe(rmsnorm(x))


def run(s):
    if s.call == "graph":
        s.graph.launch()
        return s.out
    if s.call == "block":
        _enqueue(s)
        return s.out
    if s.call == "serve":
        return s.buckets.step(s.x)
    s.layers[0].forward_host(s.x, s.y)  # y += moe(x)
    return s.y


def work(case):
    """Each picked expert's weights once per layer, the router, the rows in and out."""
    h, e, k, i, t = case["hidden"], case["experts"], case["topk"], case["inter"], case["tokens"]
    distinct = e * (1.0 - (1.0 - k / e) ** t)
    weight_bits = 8.5 if case["fmt"] == "q8" else 4.625  # a 16-bit scale per 32 weights, or 160 bits per 256
    per_layer = distinct * 3 * i * h * weight_bits / 8 + e * h * 2
    flops = case["layers"] * 2.0 * t * (k * 3 * i * h + e * h)
    return {"bytes": case["layers"] * per_layer + 2.0 * t * h * 4, "flops": flops}


def tolerance(case):
    """f32 sums (about 1e-7 each), but the SwiGLU rows are rounded to 8 bits on the way: a sum that
    differs in its last bit now and then rounds to the neighbouring value, which is what these allow."""
    return {"rel": 1e-4, "max": 4e-3}
