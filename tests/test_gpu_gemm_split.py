"""K-split prefill GEMMs: where their partial products lie.  Graphs keep their buffer, streams do not share one, a first
call may happen inside a capture, and the same call gives the same bits eager and captured."""
import pytest
import torch

import leviathan_b200 as lev
from leviathan_b200 import quant as Q
from tests import helpers as H

pytestmark = pytest.mark.gpu


def make(ctx, name, rows, cols, tokens, seed):
    w = ctx.upload(H.quantized(H.TYPES[name], seed, rows, cols), H.TYPES[name], rows, cols)
    x = torch.from_numpy(Q.normal(seed + 1, (tokens, cols), 1.0)).cuda().to(torch.bfloat16)
    return w, x


@pytest.fixture()
def ctx():
    c = lev.Context(0)   # one per test: no buffer is left by another
    yield c
    c.close()


def captured(ctx, w, x, y):
    stream, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        ctx.gemm_prefill(w, x, out=y)
    return g


@pytest.mark.parametrize("name,rows,cols,tokens", [
    ("q4_0", 2816, 1408, 32),     # a decode batch: six splits, the context's graph buffer
    ("q4_0", 13056, 4096, 16),
    ("q4_k", 512, 4096, 128),
    ("q6_k", 512, 4096, 40),      # six-bit and longer calls: a buffer per capture and stream
    ("q6_k", 512, 4096, 300),
    ("q4_0", 2816, 4096, 256),
    ("q4_k", 1024, 8192, 513),
])
def test_first_call_inside_a_capture(ctx, name, rows, cols, tokens):
    w, x = make(ctx, name, rows, cols, tokens, 71)
    y = torch.zeros((tokens, rows), device="cuda")
    g = captured(ctx, w, x, y)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ctx.gemm_prefill(w, x))
    w.free()


def test_a_captured_batch_keeps_its_buffer(ctx):
    """Longer calls after the capture, eager and captured, must not take the buffer from under the graph."""
    w, x = make(ctx, "q4_0", 2816, 4096, 32, 72)
    want = ctx.gemm_prefill(w, x)
    y = torch.zeros_like(want)
    g = captured(ctx, w, x, y)
    others = []
    for name, rows, cols, tokens in (("q6_k", 4096, 12288, 301), ("q4_0", 2816, 4096, 256), ("q4_0", 2816, 4096, 128)):
        wo, xo = make(ctx, name, rows, cols, tokens, 73)
        yo = ctx.gemm_prefill(wo, xo)
        go = captured(ctx, wo, xo, yo)
        others.append((go, wo, xo, yo))   # a graph reads and writes them
    ctx.synchronize()
    fill = torch.full((1 << 26,), float("nan"), device="cuda")   # takes what was given back, if anything was
    for _ in range(3):
        y.zero_()
        for go, *_ in others:
            go.replay()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    del fill
    for _, wo, _, _ in others:
        wo.free()
    w.free()


def test_captured_prompts_do_not_share_a_buffer(ctx):
    """Two graphs of one context replayed side by side."""
    runs = []
    for seed in (90, 91):
        w, x = make(ctx, "q6_k", 4096, 8192, 200, seed)
        want = ctx.gemm_prefill(w, x)
        y = torch.zeros_like(want)
        runs.append((w, x, want, y, captured(ctx, w, x, y), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for _ in range(4):
        for *_, g, s in runs:
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    for w, _, want, y, _, _ in runs:
        assert torch.equal(y, want)
        w.free()


def test_streams_do_not_share_a_buffer(ctx):
    """Six streams with two calls each in flight: the first have buffers of their own, the others do not split.  f32 sums
    of K products in two orders differ by at most K * 2^-23 of the sum of their magnitudes."""
    cases = [make(ctx, "q6_k", 4096, 8192, 150 + 16 * i, 80 + i) for i in range(6)]
    want, bound = [], []
    for w, x in cases:
        want.append(ctx.gemm_prefill(w, x))
        d = torch.empty((4096, 8192), device="cuda")
        ctx.dequantize(w, device_out=d)
        bound.append(8192 * 2.0 ** -23 * (x.float().abs() @ d.to(torch.bfloat16).float().abs().T))
        ctx.synchronize()
    streams = [torch.cuda.Stream() for _ in range(6)]
    torch.cuda.synchronize()
    got = [[] for _ in cases]
    for _ in range(2):
        for i, (w, x) in enumerate(cases):
            with torch.cuda.stream(streams[i]):
                got[i].append(ctx.gemm_prefill(w, x))
    torch.cuda.synchronize()
    for i in range(6):
        for y in got[i]:
            assert torch.equal(y, want[i]) if i < 3 else bool(((y - want[i]).abs() <= bound[i]).all())
    for w, _ in cases:
        w.free()
