"""The per-token calls through the native host layer and through ctypes: the same launches, the same bits."""
import pytest
import torch

import leviathan_b200 as lev
from leviathan_b200 import _lib as L
from leviathan_b200 import quant as Q

pytestmark = pytest.mark.gpu


def calls(ctx, g):
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    w = ctx.upload(Q.quantize(Q.GGML_Q4_0, r(64, 512) * 0.02), Q.GGML_Q4_0, 64, 512)
    x, nw, res = r(3, 512), r(512), r(3, 64)
    yield ctx.matvec(w, x)
    yield ctx.matvec_fused(w, x, "rmsnorm", nw, 1e-5, residual=res, alpha=-0.5)
    yield ctx.matvec_fused(w, r(1024), "gelu_up")
    yield from ctx.matvec_chain([dict(w=w, x=x[0], out=torch.empty(64, device="cuda")),
                                 dict(w=w, x=x[1], out=torch.empty(64, device="cuda"), prologue="rmsnorm", norm_weight=nw)])
    yield ctx.rmsnorm(x, nw, 1e-6)
    yield from ctx.rmsnorm(x, None, 1e-6, want_inverse=True)
    yield ctx.axpy(0.25, x, r(3, 512))
    xb = ctx.act_bf16(r(32, 512))
    yield xb
    yield ctx.gemm_prefill(w, xb)
    rw, gu, dn = r(8, 96), Q.quantize_q4_0(r(8 * 64, 96) * 0.02), Q.quantize_q4_0(r(8 * 96, 32) * 0.02)
    mw = ctx.moe_upload(rw, gu, dn, 8, 96, 32)
    xm = r(5, 96)
    yield from ctx.moe_layer(mw, xm, 3, want_routing=True)
    yield ctx.moe_layer_residual(mw, xm, 3, r(5, 96), 0.5)
    cache = lev.PagedKV(8, 16, 2, 128, 2, 4)
    slot = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    for p in range(3):
        for s in range(2):
            cache.ensure(s, p)
        pos = torch.full((2,), p, dtype=torch.int32, device="cuda")
        ctx.kv_append(cache, slot, pos, r(2, 2, 128), r(2, 2, 128))
        yield ctx.attn_decode(cache, slot, pos, r(2, 8, 128), 0, 0.125)


def test_native_and_ctypes_give_the_same_bits():
    out = []
    for form in (L.host(), L._CtypesHost(L.load())):
        ctx = lev.Context(0)
        ctx.host = form
        got = [y.clone() for y in calls(ctx, torch.Generator(device="cuda").manual_seed(3))]
        ctx.synchronize()
        out.append((got, ctx.launch_count()))
    (a, la), (b, lb) = out
    assert la == lb and len(a) == len(b) == 18
    for u, v in zip(a, b):
        assert torch.equal(u, v) and bool(torch.isfinite(u.float()).all())
