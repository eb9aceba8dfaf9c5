"""The grouped dequant-GEMM of prefill-sized MoE calls (k_moe_gemm) at the edges of its tiles, stages and jobs, every
pair against the experts in f64."""
import numpy as np
import pytest
import torch

import leviathan_b200 as lev
from leviathan_b200 import quant as Q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lev.Context(0)
    yield c
    c.close()


class Layer:
    def __init__(self, ctx, experts, hidden, inter, seed, edit=None):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.dims = experts, hidden, inter
        self.gu = Q.quantize_q4_0(torch.randn((experts * 2 * inter, hidden), generator=g, device="cuda") * 0.02).cpu().numpy()
        self.dn = Q.quantize_q4_0(torch.randn((experts * hidden, inter), generator=g, device="cuda") * 0.02).cpu().numpy()
        if edit:
            edit(self.gu, self.dn)
        self.rw = np.zeros((experts, hidden), np.float32)
        self.mw = ctx.moe_upload(self.rw, self.gu, self.dn, experts, hidden, inter)

    def weights(self):
        e, h, i = self.dims
        f64 = lambda b, r, c: torch.from_numpy(O.dequantize_rows(Q.GGML_Q4_0, b, r, c)).cuda().double()
        return f64(self.gu, e * 2 * i, h).view(e, 2 * i, h), f64(self.dn, e * h, i).view(e, h, i)


def reference(layer, x, idx):
    """(y, bound of y, act, bound of act) per pair in f64.  Operands are rounded once to 11 bits (half a unit: 2^-11 of the
    value; activations at least 2^-39 of their row's largest), products are exact and K of them are added in f32.  |gelu'|
    is at most 1.13."""
    gu, dn = layer.weights()
    e, h, i = layer.dims
    t, k = idx.shape
    x64, flat = x.double(), idx.reshape(-1).long()
    act = torch.zeros((t * k, i), dtype=torch.float64, device="cuda")
    act_b, y, y_b = torch.zeros_like(act), torch.zeros((t * k, h), dtype=torch.float64, device="cuda"), None
    y_b = torch.zeros_like(y)

    def dot(v, v_err, w):
        rel = 2.0 ** -10 + 2.0 ** -21 + v.shape[1] * 2.0 ** -24
        lost = 2.0 ** -38 * v.abs().amax(1, keepdim=True) * w.abs().sum(1)
        return v @ w.T, rel * ((v.abs() + v_err) @ w.abs().T) + v_err @ w.abs().T + lost

    for ex in range(e):
        p = (flat == ex).nonzero()[:, 0]
        if not len(p):
            continue
        v = x64[p // k]
        g, g_e = dot(v, torch.zeros_like(v), gu[ex, :i])
        u, u_e = dot(v, torch.zeros_like(v), gu[ex, i:])
        gl = torch.nn.functional.gelu(g, approximate="tanh")
        act[p] = gl * u
        act_b[p] = 1.13 * g_e * (u.abs() + u_e) + gl.abs() * u_e + 2.0 ** -20 * (gl * u).abs() + 1e-37
        y[p], y_b[p] = dot(act[p], act_b[p], dn[ex])
    return y.view(t, k, h), y_b.view(t, k, h), act.view(t, k, i), act_b.view(t, k, i)


def routing(rng, tokens, top_k, experts, crowd=0):
    """top_k different experts per token; the first `crowd` tokens all have expert 1."""
    idx = np.stack([rng.permutation(experts)[:top_k] for _ in range(tokens)]).astype(np.int32)
    for t in range(crowd):
        if 1 not in idx[t]:
            idx[t, t % top_k] = 1
    return torch.from_numpy(idx).cuda()


def check(ctx, layer, x, idx, times=1):
    want, bound, _, _ = reference(layer, x, idx)
    ctx.moe_experts(layer.mw, x, idx)
    for _ in range(times):
        y = ctx.moe_experts(layer.mw, x, idx)
        ctx.synchronize()
        assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())


@pytest.mark.parametrize("hidden,inter", [(1152, 320), (1408, 384), (2176, 640), (640, 896), (384, 128), (896, 96)])
def test_odd_numbers_of_stages(ctx, hidden, inter):
    """Two chunks of 64 columns make a stage of the 64-token jobs: with an odd number of stages a tile ends in a K-step of
    one stage, and a decode team passes over K-steps of the raw ring."""
    rng = np.random.default_rng(hidden)
    layer = Layer(ctx, 32, hidden, inter, hidden + inter)
    x = torch.from_numpy(Q.normal(hidden, (260, hidden), 1.0)).cuda()
    check(ctx, layer, x, routing(rng, 260, 4, 32), times=8)
    layer.mw.free()


@pytest.mark.parametrize("experts,hidden,inter,top_k,tokens", [(8, 256, 96, 4, 160), (16, 512, 128, 8, 64)])
def test_activations_off_a_16_byte_boundary(ctx, experts, hidden, inter, top_k, tokens):
    """A view that starts one float into its buffer, at 512 and 640 pairs: the job-list kernel does not take such rows, so
    the grouped GEMM does."""
    rng = np.random.default_rng(tokens)
    layer = Layer(ctx, experts, hidden, inter, 7)
    buf = torch.from_numpy(Q.normal(8, (tokens * hidden + 1,), 1.0)).cuda()
    x = buf[1:].view(tokens, hidden)
    assert x.data_ptr() % 16 == 4
    idx = routing(rng, tokens, top_k, experts)
    check(ctx, layer, x, idx)
    out = ctx.moe_layer(layer.mw, x, top_k)
    ref = ctx.moe_layer(layer.mw, x.clone(), top_k)
    ctx.synchronize()
    assert float((out - ref).norm() / ref.norm()) < 2e-3   # the aligned call may take the job-list kernel
    layer.mw.free()


@pytest.mark.parametrize("first,count", [(0, 8), (24, 8), (12, 4)])
def test_resident_experts_only(ctx, first, count):
    """A rank's share of the experts at a prefill-sized call: its pairs, nothing else, and the jobs are sized by an
    expert's share of all pairs."""
    rng = np.random.default_rng(first)
    e, h, i = 32, 640, 192
    layer = Layer(ctx, e, h, i, 300 + first)
    gs, ds = 2 * i * (h // 32) * 18, h * (i // 32) * 18
    part = ctx.moe_upload(layer.rw, layer.gu[first * gs:(first + count) * gs], layer.dn[first * ds:(first + count) * ds], e, h, i,
                          local_first=first, local_count=count)
    x = torch.from_numpy(Q.normal(31, (256, h), 1.0)).cuda()
    idx = routing(rng, 256, 4, e)
    mine = ((idx >= first) & (idx < first + count))
    y = ctx.moe_experts(part, x, idx)
    ctx.synchronize()
    want, bound, _, _ = reference(layer, x, idx)
    assert bool(((y.double() - want).abs() <= bound)[mine].all())
    part.free()
    layer.mw.free()


@pytest.mark.parametrize("experts,hidden,inter,top_k,tokens,crowd", [
    (8, 1056, 96, 2, 600, 0),       # 256-token jobs (over 40 pairs an expert); hidden and inter with half chunks of K and
    (8, 1056, 96, 2, 600, 590),     # partly filled row tiles; an expert with three jobs, the last ragged
    (4, 256, 32, 1, 1030, 0),       # one chunk of K in the down product: teams without work
    (4, 64, 32, 2, 520, 513),       # one chunk in both, a last job of one token
    (32, 1056, 96, 4, 256, 200),    # 64-token jobs, several of one expert
    (32, 96, 544, 4, 260, 129),
    (64, 192, 224, 8, 130, 0),
])
def test_jobs_tiles_and_remainders(ctx, experts, hidden, inter, top_k, tokens, crowd):
    rng = np.random.default_rng(hidden + crowd)
    layer = Layer(ctx, experts, hidden, inter, hidden + inter + crowd)
    x = torch.from_numpy(Q.normal(tokens, (tokens, hidden), 1.0)).cuda()
    idx = routing(rng, tokens, top_k, experts, crowd)
    want, bound, act, act_b = reference(layer, x, idx)
    y, a = ctx.moe_experts(layer.mw, x, idx, want_act=True)
    ctx.synchronize()
    assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())
    assert bool(((a.double() - act).abs() <= act_b).all()), float(((a.double() - act).abs() / act_b).max())
    assert torch.equal(y, ctx.moe_experts(layer.mw, x, idx))
    layer.mw.free()


def test_rows_of_any_magnitude(ctx):
    """A row of activations is scaled by a power of two of its own: zeros, far below and above the f16 range, and one with an
    infinity, whose token alone is not finite."""
    rng = np.random.default_rng(5)
    layer = Layer(ctx, 32, 1152, 128, 55)
    x = torch.from_numpy(Q.normal(56, (256, 1152), 1.0)).cuda()
    x[3], x[4], x[5], x[6] = 0.0, x[4] * 1e-30, x[5] * 1e9, x[6] * 1e-6
    x[7, 100] = 3e4
    x[200, 17] = float("inf")
    x[201, 1151] = float("nan")
    idx = routing(rng, 256, 4, 32)
    y = ctx.moe_experts(layer.mw, x, idx)
    ctx.synchronize()
    bad = torch.zeros(256, dtype=torch.bool, device="cuda")
    bad[[200, 201]] = True
    assert not bool(torch.isfinite(y[bad]).any())
    clean = x.clone()
    clean[bad] = 0.0
    want, bound, _, _ = reference(layer, clean, idx)
    assert bool(((y.double() - want).abs() <= bound)[~bad].all())
    assert bool((y[3] == 0).all())
    layer.mw.free()


def test_scales_beyond_f16_products_take_the_f32_forms(ctx):
    """A block scale of 65504: d * (q - 8) leaves the f16 range, so the layer keeps to the kernels with f32 scales."""
    def edit(gu, dn):
        dn[0:2] = np.array([0xFF, 0x7B], np.uint8)                      # expert 0, row 0, block 0
        dn[18 * 4 * 10:18 * 4 * 10 + 2] = np.array([0xFF, 0xFB], np.uint8)   # row 10: the negative one

    rng = np.random.default_rng(6)
    layer = Layer(ctx, 32, 256, 128, 66, edit)
    x = torch.from_numpy(Q.normal(67, (256, 256), 1.0)).cuda()
    idx = routing(rng, 256, 4, 32)
    y = ctx.moe_experts(layer.mw, x, idx)
    ctx.synchronize()
    want, bound, _, _ = reference(layer, x, idx)
    assert bool(torch.isfinite(y).all()) and bool(((y.double() - want).abs() <= bound).all())
    assert float((y.double() - want).norm() / want.norm()) < 1e-4
    layer.mw.free()
