"""Prefill dequant-GEMM against the rounded-operand f64 oracle
(rust/crates/lev-cli/src/main.rs:1201-1275), through the C ABI."""
import numpy as np
import pytest
import torch

import leviathan_b200 as lev
from leviathan_b200 import quant as Q
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

# north-star pass bar for bf16 tensor-core prefill, and the reference's own f16 gate
PASS_TOL, REPORT_TOL = 2e-2, 1e-3


@pytest.fixture(scope="module")
def ctx():
    c = lev.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name,rows,cols,tokens", [
    ("q4_k", 256, 1024, 64), ("q4_k", 80, 512, 37), ("q6_k", 128, 768, 70), ("q4_0", 96, 704, 5), ("q4_0", 64, 2816, 128),
    # several row tiles with a ragged last one, two token tiles (256 + 44)
    ("q4_k", 400, 512, 300), ("q6_k", 360, 256, 130),
    # decode batches against tensors of a few row tiles: raw bytes staged in shared memory, K split over the grid
    # (11 groups of 256 columns over 8 splits; 8 groups over 8; a ragged last row tile; one token)
    ("q4_0", 528, 2816, 32), ("q4_k", 352, 2048, 32), ("q4_k", 200, 1024, 128), ("q4_0", 176, 512, 1),
])
def test_gemm_matches_rounded_operand_oracle(ctx, name, rows, cols, tokens):
    t = H.TYPES[name]
    w = H.quantized(t, 21, rows, cols)
    x = Q.normal(22, (tokens, cols), 1.0)
    wh = ctx.upload(w, t, rows, cols)
    xb = ctx.act_bf16(torch.from_numpy(x).cuda())
    # the conversion is round-to-nearest-even like torch's
    assert torch.equal(xb, torch.from_numpy(x).cuda().to(torch.bfloat16))
    buf, view = H.guarded(tokens * rows)
    y = ctx.gemm_prefill(wh, xb, out=view.view(tokens, rows))
    torch.cuda.synchronize()
    assert H.guards_intact(buf, tokens * rows)
    y = y.cpu().numpy()
    step = 13 if rows > 64 else 1  # every 13th row x all tokens, like the reference's gate
    ref = O.gemm_rounded_f64(t, w, rows, cols, x, "bf16", 0, step)
    err = O.max_rel_err(y[:, ::step], ref)
    assert err < REPORT_TOL and err < PASS_TOL, (name, err)
    y2 = ctx.gemm_prefill(wh, xb).cpu().numpy()
    assert np.array_equal(y.view(np.uint32), y2.view(np.uint32))
    wh.free()


def test_gemm_rejections(ctx):
    w = H.quantized(Q.GGML_Q4_K, 1, 64, 256)
    wh = ctx.upload(w, Q.GGML_Q4_K, 64, 256)
    with pytest.raises(lev.LevError) as e:
        ctx.lib.lev_gemm_prefill.restype  # keep the binding imported
        ctx._check(ctx.lib.lev_gemm_prefill(ctx.handle, wh.handle, 1, 0, 1, 0))
    assert e.value.name == "badDimensions"
    wh.free()


@pytest.mark.parametrize("name", ["q4_0", "q4_k", "q6_k"])
@pytest.mark.parametrize("rows,cols,tokens", [
    (16, 256, 17),       # one 16-row tile of eight, a second N step of 16
    (272, 1280, 129),    # first size of the CTA pairs: the last pair's second CTA has no rows; five K-steps of 256
    (250, 768, 288),     # two MMAs side by side, a ragged last row
    (144, 512, 513),     # a second token tile
])
def test_gemm_tile_edges(ctx, name, rows, cols, tokens):
    """Edges of the row tiles (16, 128, 256), of N (16 / 32, 256, 512) and of the K-steps, against the rounded operands
    in f64.  An f32 sum of K products differs from it by at most K * 2^-24 of the sum of their magnitudes."""
    t = H.TYPES[name]
    wh = ctx.upload(H.quantized(t, 23, rows, cols), t, rows, cols)
    w = torch.empty((rows, cols), device="cuda")
    ctx.dequantize(wh, device_out=w)
    xb = torch.from_numpy(Q.normal(24, (tokens, cols), 1.0)).cuda().to(torch.bfloat16)
    y = ctx.gemm_prefill(wh, xb)
    ctx.synchronize()
    wb = w.to(torch.bfloat16).double()
    ref, bound = xb.double() @ wb.T, cols * 2.0 ** -24 * (xb.double().abs() @ wb.abs().T)
    assert bool(((y.double() - ref).abs() <= bound).all()), float(((y.double() - ref).abs() - bound).max())
    assert torch.equal(y, ctx.gemm_prefill(wh, xb))
    wh.free()


def test_prompt_call_captured_first(ctx):
    """A prompt-sized call whose first use is inside a capture: no work buffer may be needed there."""
    t = H.TYPES["q6_k"]
    fresh = lev.Context(0)
    wh = fresh.upload(H.quantized(t, 61, 512, 4096), t, 512, 4096)
    xb = torch.from_numpy(Q.normal(62, (300, 4096), 1.0)).cuda().to(torch.bfloat16)
    y = torch.zeros((300, 512), device="cuda")
    torch.cuda.synchronize()
    stream, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        fresh.gemm_prefill(wh, xb, out=y)
    g.replay()
    torch.cuda.synchronize()
    ref = fresh.gemm_prefill(wh, xb)   # may split K: another order of the same f32 sums
    fresh.synchronize()
    assert float((y - ref).norm() / ref.norm()) < 4096 * 2.0 ** -24
    wh.free()
    fresh.close()
