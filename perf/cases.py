"""Timing cases: the calls a host of this package makes, over the sizes it makes them at.

Six kinds of pass, each through the public Python layer on device tensors unless it says otherwise:

  matvec   Context.matvec: one resident tensor, one to eight activation columns
  ffn      Context.chain_submit of a prepared list: gate, up and down of a dense FFN at one column, either as
           independent products (device or pinned host buffers) or as the dependent block
           norm -> gate, up -> gelu-up -> down -> residual
  prefill  Context.act_bf16 + Context.gemm_prefill: f32 activations of a prompt or a wide decode batch
  moe      Context.moe_layer_residual: router, top-k, grouped experts, combine and the residual step
  attn     Context.kv_append + Context.attn_decode over a paged cache, sequences of different lengths
  decode   SyntheticDecoder: a captured decode step of a whole model, token ids handed in for each step
"""
import math

import numpy as np
import torch

import leviathan_b200 as lev
from leviathan_b200 import quant as Q
from leviathan_b200.decoder import DecoderConfig, SyntheticDecoder

TYPES = {"q4_0": Q.GGML_Q4_0, "q4_k": Q.GGML_Q4_K, "q6_k": Q.GGML_Q6_K}
BLOCK = {"q4_0": (32, 18), "q4_k": (256, 144), "q6_k": (256, 210)}
DEV = "cuda"


def listed():
    return [
        # the k or v projection of one decoded token: the smallest call of a decode loop
        dict(name="matvec_kv_proj", kind="matvec", type="q4_0", rows=2048, cols=2816, n=1),
        # an FFN tensor for a handful of sequences decoded together
        dict(name="matvec_six_columns", kind="matvec", type="q4_k", rows=12288, cols=4096, n=6),
        # a dense FFN's three products at batch 1 in one submission
        dict(name="ffn_list", kind="ffn", inter=12288, hidden=4096, block=False, host=False),
        # the same from a host whose activations live in pinned host memory
        dict(name="ffn_list_host", kind="ffn", inter=12288, hidden=4096, block=False, host=True),
        # a prompt of 512 tokens through an FFN tensor
        dict(name="prefill_512", kind="prefill", type="q4_k", rows=12288, cols=4096, tokens=512),
        # a prompt of odd length through the six-bit down projection
        dict(name="prefill_ragged_q6k", kind="prefill", type="q6_k", rows=4096, cols=12288, tokens=301),
        # the routed experts of one decoded token
        dict(name="moe_1", kind="moe", experts=128, top_k=8, hidden=2816, inter=704, tokens=1),
        # of a decode batch
        dict(name="moe_48", kind="moe", experts=128, top_k=8, hidden=2816, inter=704, tokens=48),
        # of a prompt
        dict(name="moe_512", kind="moe", experts=128, top_k=8, hidden=2816, inter=704, tokens=512),
        # one sequence's attention at a context of 4096
        dict(name="attn_one_sequence", kind="attn", q_heads=16, kv_heads=8, head_dim=256, seqs=1, positions=4096, kv="f16", window=0),
        # a decoded token of the whole synthetic model
        dict(name="decode_batch_1", kind="decode", batch=1, layers=30, positions=4096, hidden=2816, experts=128, inter=704, vocab=262144),
        # a decoded token for 32 sequences on twelve of its layers
        dict(name="decode_batch_32", kind="decode", batch=32, layers=12, positions=4096, hidden=2816, experts=128, inter=704, vocab=262144),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["matvec", "ffn", "prefill", "moe", "attn", "decode"])
    t = rng.choice(["q4_0", "q4_k", "q6_k"])
    step = 32 if t == "q4_0" else 256
    if kind == "matvec":
        n = rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8])
        return dict(kind=kind, type=t, rows=_log(rng, 128, 65536), cols=_log(rng, 256, 12288, step), n=n)
    if kind == "ffn":
        block = rng.random() < 0.5
        return dict(kind=kind, inter=_log(rng, 1024, 16384, 256), hidden=_log(rng, 1024, 8192, 256), block=block,
                    host=not block and rng.random() < 0.5)
    if kind == "prefill":
        # 64 columns are the tensor-core kernels' step: the 4-bit format with small blocks has odd multiples of 32 too
        return dict(kind=kind, type=t, rows=_log(rng, 256, 16384), cols=_log(rng, 512, 12288, step), tokens=_log(rng, 9, 2048))
    if kind == "moe":
        experts = rng.choice([16, 32, 64, 128])
        return dict(kind=kind, experts=experts, top_k=rng.choice([1, 2, 4, 6, 8]), hidden=_log(rng, 1024, 4096, 64),
                    inter=_log(rng, 256, 1536, 32), tokens=_log(rng, 1, 1024))
    if kind == "attn":
        qh, kvh, hd = rng.choice([(16, 8, 256), (32, 8, 128), (16, 16, 128), (8, 2, 256)])
        seqs = _log(rng, 1, 48)
        return dict(kind=kind, q_heads=qh, kv_heads=kvh, head_dim=hd, seqs=seqs, positions=_log(rng, 64, 8192 if seqs <= 16 else 4096),
                    kv=rng.choice(["f16", "f16", "f32"]), window=rng.choice([0, 0, 1024]))
    return dict(kind=kind, batch=_log(rng, 1, 32), layers=rng.randint(2, 6), positions=_log(rng, 256, 4096),
                hidden=256 * rng.randint(4, 11), experts=rng.choice([32, 64, 128]), inter=64 * rng.randint(4, 11),
                vocab=_log(rng, 32768, 262144, 1024))


# ---- what a program has in hand before the call ----
_ctx = None
_stream = None


def _decode_stream():
    """One stream for every captured step, as one serving loop has: steps run one after another."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _context():
    global _ctx
    if _ctx is None:
        _ctx = lev.Context(0)
    return _ctx


class State:
    """Inputs and resident handles of one case; the device copies of the weights go when it goes."""

    def __init__(self, case, **kw):
        self.case = case
        self.owned = []
        self.__dict__.update(kw)

    def __del__(self):
        for o in reversed(self.owned):
            try:
                o()
            except Exception:
                pass


def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((seed * 1000003 + salt) & 0x7FFFFFFFFFFF)


def _weights(s, ctx, t, rows, cols, g):
    """N(0, 0.02) weights, encoded and uploaded."""
    parts = []
    slab = max(1, (1 << 26) // cols)
    for r in range(0, rows, slab):
        n = min(slab, rows - r)
        parts.append(Q.quantize(TYPES[t], torch.randn((n, cols), generator=g, device=DEV) * 0.02))
    w = ctx.upload(torch.cat(parts), TYPES[t], rows, cols)
    s.owned.append(w.free)
    return w


def prepare(case, seed):
    kind, s = case["kind"], State(case)
    g = _gen(seed)
    if kind == "decode":
        # a context of its own: the captured step holds addresses of the context's work buffers
        s.ctx = lev.Context(0)
        s.owned.append(s.ctx.close)
        s.stream = _decode_stream()
        cfg = DecoderConfig(hidden=case["hidden"], layers=case["layers"], experts=case["experts"], expert_inter=case["inter"],
                            vocab=case["vocab"], positions=case["positions"], seed=0x4C455649 ^ (seed << 24))
        with torch.cuda.stream(s.stream):
            s.dec = SyntheticDecoder(s.ctx, cfg, batch=case["batch"])
            s.owned.append(s.dec.free)
            s.ids = torch.randint(0, case["vocab"], (case["batch"],), generator=g, device=DEV).to(torch.int32)
            s.dec.tok.copy_(s.ids)
            s.dec.capture()
            s.dec.tok.copy_(s.ids)
        s.stream.synchronize()
        return s
    s.ctx = ctx = _context()
    if kind == "matvec":
        s.w = _weights(s, ctx, case["type"], case["rows"], case["cols"], g)
        s.x = torch.randn((case["n"], case["cols"]), generator=g, device=DEV)
    elif kind == "ffn":
        I, H = case["inter"], case["hidden"]
        gate, up = _weights(s, ctx, "q4_k", I, H, g), _weights(s, ctx, "q4_k", I, H, g)
        down = _weights(s, ctx, "q6_k", H, I, g)
        x, a = torch.randn(H, generator=g, device=DEV), torch.randn(I, generator=g, device=DEV)
        if case["block"]:
            s.gu, s.y = torch.empty(2 * I, device=DEV), torch.empty(H, device=DEV)
            norm = 1.0 + 0.02 * torch.randn(H, generator=g, device=DEV)
            ops = [dict(w=gate, x=x, out=s.gu[:I], prologue="rmsnorm", norm_weight=norm),
                   dict(w=up, x=x, out=s.gu[I:], prologue="rmsnorm", norm_weight=norm),
                   dict(w=down, x=s.gu, out=s.y, prologue="gelu_up", residual=x, alpha=1.0)]
            s.outs = [s.gu, s.y]
        elif case["host"]:
            def pinned(n, src=None):
                t = torch.empty(n, pin_memory=True)
                if src is not None:
                    t.copy_(src)
                s.__dict__.setdefault("keep", []).append(t)
                return t.numpy()

            hx, ha = pinned(H, x), pinned(I, a)
            ops = [dict(w=gate, x=hx, out=pinned(I)), dict(w=up, x=hx, out=pinned(I)), dict(w=down, x=ha, out=pinned(H))]
            s.outs = [o["out"] for o in ops]
        else:
            ops = [dict(w=gate, x=x, out=torch.empty(I, device=DEV)), dict(w=up, x=x, out=torch.empty(I, device=DEV)),
                   dict(w=down, x=a, out=torch.empty(H, device=DEV))]
            s.outs = [o["out"] for o in ops]
        s.list = ctx.chain_prepare(ops)
    elif kind == "prefill":
        s.w = _weights(s, ctx, case["type"], case["rows"], case["cols"], g)
        s.x = torch.randn((case["tokens"], case["cols"]), generator=g, device=DEV)
    elif kind == "moe":
        E, H, I = case["experts"], case["hidden"], case["inter"]
        gu, dn = [], []
        for e in range(0, E, 16):
            n = min(16, E - e)
            gu.append(Q.quantize(Q.GGML_Q4_0, torch.randn((n * 2 * I, H), generator=g, device=DEV) * 0.02))
            dn.append(Q.quantize(Q.GGML_Q4_0, torch.randn((n * H, I), generator=g, device=DEV) * 0.02))
        router = torch.randn((E, H), generator=g, device=DEV) * 0.02
        s.w = ctx.moe_upload(router, torch.cat(gu), torch.cat(dn), E, H, I)
        s.owned.append(s.w.free)
        s.x = torch.randn((case["tokens"], H), generator=g, device=DEV)
        s.res = torch.randn((case["tokens"], H), generator=g, device=DEV)
        s.out = torch.empty_like(s.res)
    elif kind == "attn":
        n, P, page = case["seqs"], case["positions"], 16
        per = (P + page - 1) // page
        s.cache = lev.PagedKV(n * per + 1, page, case["kv_heads"], case["head_dim"], slots=n, max_blocks=per, dtype=case["kv"], device=DEV)
        # sequences of one batch differ in length: between three quarters of the context and all of it
        lens = [P] + [P - int(v) for v in np.random.RandomState(seed & 0x7FFFFFFF).randint(0, max(1, P // 4), n - 1)]
        for q in range(n):
            s.cache.ensure(q, lens[q] - 1)
        s.cache.k.normal_(generator=g)
        s.cache.v.normal_(generator=g)
        s.slot = torch.arange(n, dtype=torch.int32, device=DEV)
        s.pos = torch.tensor([v - 1 for v in lens], dtype=torch.int32, device=DEV)
        s.q = torch.randn((n, case["q_heads"], case["head_dim"]), generator=g, device=DEV)
        s.k = torch.randn((n, case["kv_heads"], case["head_dim"]), generator=g, device=DEV)
        s.v = torch.randn((n, case["kv_heads"], case["head_dim"]), generator=g, device=DEV)
        s.scale = 1.0 / math.sqrt(case["head_dim"])
    return s


def run(s):
    kind, ctx = s.case["kind"], s.ctx
    if kind == "matvec":
        return ctx.matvec(s.w, s.x)
    if kind == "ffn":
        ctx.chain_submit(s.list)
        return s.outs
    if kind == "prefill":
        return ctx.gemm_prefill(s.w, ctx.act_bf16(s.x))
    if kind == "moe":
        return ctx.moe_layer_residual(s.w, s.x, s.case["top_k"], s.res, 1.0, out=s.out)
    if kind == "attn":
        ctx.kv_append(s.cache, s.slot, s.pos, s.k, s.v)
        return ctx.attn_decode(s.cache, s.slot, s.pos, s.q, s.case["window"], s.scale)
    with torch.cuda.stream(s.stream):
        s.dec.tok.copy_(s.ids)  # the scheduler's token ids of this step
        s.dec.replay()
    return {"token": s.dec.tok, "logits": s.dec.logits}


# ---- what a pass cannot do without ----
def _gguf(t, rows, cols):
    return rows * (cols // BLOCK[t][0]) * BLOCK[t][1]


def _distinct(experts, top_k, tokens):
    """Experts that `tokens` independent choices of top_k touch, on average."""
    return experts * (1.0 - (1.0 - top_k / experts) ** tokens)


def _moe_work(E, k, H, I, T):
    expert = _gguf("q4_0", 2 * I, H) + _gguf("q4_0", H, I)
    return dict(bytes=_distinct(E, k, T) * expert + 4 * E * H + 12 * T * H, flops=2.0 * T * (k * 3 * H * I + E * H))


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "prefill"):
        n = case["n"] if kind == "matvec" else case["tokens"]
        return dict(bytes=_gguf(case["type"], case["rows"], case["cols"]) + 4 * n * (case["rows"] + case["cols"]),
                    flops=2.0 * n * case["rows"] * case["cols"])
    if kind == "ffn":
        I, H = case["inter"], case["hidden"]
        return dict(bytes=2 * _gguf("q4_k", I, H) + _gguf("q6_k", H, I) + 4 * (3 * I + 2 * H), flops=6.0 * I * H)
    if kind == "moe":
        return _moe_work(case["experts"], case["top_k"], case["hidden"], case["inter"], case["tokens"])
    if kind == "attn":
        n, live = case["seqs"], min(case["positions"], case["window"] or case["positions"])
        mean = live if case["window"] else case["positions"] * (1 + 7 * (n - 1) / 8) / n
        row = case["kv_heads"] * case["head_dim"]
        return dict(bytes=n * (2 * mean * row * (2 if case["kv"] == "f16" else 4) + 8 * case["q_heads"] * case["head_dim"] + 8 * row),
                    flops=4.0 * n * mean * case["q_heads"] * case["head_dim"])
    B, L, H, P = case["batch"], case["layers"], case["hidden"], case["positions"]
    qw, kw = 4096, 2048  # 16 query and 8 key / value heads of 256
    proj = _gguf("q4_0", qw + 2 * kw, H) + _gguf("q4_0", H, qw)
    moe = _moe_work(case["experts"], 8, H, case["inter"], B)
    head = _gguf("q6_k", case["vocab"], H)
    return dict(bytes=L * (proj + moe["bytes"] + B * 2 * P * kw * 2) + head + 4 * B * case["vocab"],
                flops=L * (2.0 * B * H * (2 * qw + 2 * kw) + moe["flops"] + 4.0 * B * P * qw) + 2.0 * B * case["vocab"] * H)


def tolerance(case):
    kind = case["kind"]
    if kind in ("matvec", "attn") or (kind == "ffn" and not case["block"]):
        return {"rel": 1e-5}  # f32 activations, f32 sums
    if kind == "ffn":
        return {"rel": 2e-5}  # two products behind one another
    if kind == "prefill":
        return {"rel": 4e-3}  # operands rounded to bf16
    if kind == "moe":
        # from 512 token-slot pairs on the operands are rounded to bf16, the activations between the two products too
        return {"rel": 2e-5 if case["tokens"] * case["top_k"] < 512 else 6e-3}
    if case["batch"] < 16:
        return {"rel": 1e-3}  # f32 arithmetic, K and V rounded to f16 in every layer
    # bf16 projections layer after layer; a near-tie of two experts or two tokens may fall the other way
    return {"rel": 2e-2, "differ": 0.07}
