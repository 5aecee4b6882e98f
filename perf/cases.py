"""The work that is measured: what a user of the library has it do, over the sizes that this repository's configurations name.

Seven kinds, each through the package's public entry points:

  gemv       one quantised matrix-vector product, called as an operator (a projection, the head of a model)
  token      the matrix products of one decoding step of a dense model, recorded once as a command list and replayed, as a
             serving loop does: q | k | v, output projection, gate | up with SiLU, down, head; for 1 or 2..8 sequences
  moe        a mixture-of-experts layer in 32-bit arithmetic (decoding: one to a few hundred tokens)
  experts    the same layer on the tensor cores in bf16 for a routing that is given (prefill; popularity of experts as Zipf's law)
  decode     whole call of the OLMoE-shaped decoder: a short prompt token by token, logits of its last position
  rows       a product of bf16 weights with many rows of activations (prefill of the layered decoders)
  attention  causal attention of a prefill pass over the f16 cache
"""
import math

import numpy as np
import torch

import runit_mac_b200 as R

BLOCK = {"q8_0": (32, 34), "q4_0": (32, 18), "q4k": (256, 144), "q5_0": (32, 22), "q5k": (256, 176), "q6k": (256, 210)}
FMT = {"q8_0": R.FMT_Q8_0, "q4_0": R.FMT_Q4_0, "q4k": R.FMT_Q4K, "q5_0": R.FMT_Q5_0, "q5k": R.FMT_Q5K, "q6k": R.FMT_Q6K}


def _token(fmt, batch, hidden, q_dim, kv_dim, ff, vocab, layers):
    return dict(kind="token", fmt=fmt, batch=batch, hidden=hidden, q_dim=q_dim, kv_dim=kv_dim, ff=ff, vocab=vocab, layers=layers)


def listed():
    return [
        # the smallest call: the output projection of a 0.5B model with its residual, not recorded
        dict(kind="gemv", name="o-proj q8_0 896", fmt="q8_0", m=896, k=896, add=True),
        # a decoding step of a small model on a device: many launches of 1-5 MB each
        dict(_token("q8_0", 1, 896, 896, 128, 4864, 151936, 24), name="token q8_0 0.5B"),
        # a decoding step of a 7B model for one user (a third of its layers, and the head)
        dict(_token("q4k", 1, 3584, 3584, 512, 18944, 152064, 8), name="token q4k 7B"),
        # the same for eight users at once
        dict(_token("q4k", 8, 3584, 3584, 512, 18944, 152064, 8), name="token q4k 7B x8"),
        # four users, the older 4-bit format
        dict(_token("q4_0", 4, 3584, 3584, 512, 18944, 152064, 4), name="token q4_0 7B x4"),
        # the head of a mixed-format file, which keeps it in 6 bits
        dict(kind="gemv", name="head q6k 7B", fmt="q6k", m=152064, k=3584, add=False),
        # an OLMoE-1B-7B layer while a few users decode
        dict(kind="moe", name="moe 16 tokens", T=16, h=2048, ff=1024, E=64, top=8),
        # the same layer for a large batch, or a short prompt, in 32-bit arithmetic
        dict(kind="moe", name="moe 256 tokens", T=256, h=2048, ff=1024, E=64, top=8),
        # prefill of a Qwen3-MoE-shaped block
        dict(kind="experts", name="experts bf16 4096", T=4096, h=2048, ff=768, E=128, top=8),
        # one user's OLMoE-shaped decoding, launches and dependent steps
        dict(kind="decode", name="decode olmoe", n=12, layers=6, hidden=2048, heads=16, vocab=50304, E=64, top=8, ff=1024),
        # up projection of a layered decoder's prefill
        dict(kind="rows", name="up relu2 2048", T=2048, m=8192, k=2048, epi="relu2"),
        # attention of a 2048-token prompt
        dict(kind="attention", name="attention 2048", T=2048, start=0, heads=16, kv_heads=16, hd=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "token", "token", "token", "moe", "moe", "experts", "decode", "rows", "attention"])
    if kind == "gemv":
        fmt = rng.choice(["q8_0", "q4_0", "q4k", "q5_0", "q5k", "q6k", "q6k"])
        k = BLOCK[fmt][0] * _log(rng, 512 // BLOCK[fmt][0], 18944 // BLOCK[fmt][0])
        return dict(kind=kind, fmt=fmt, m=_log(rng, 64, max(64, min(152064, 500_000_000 // k))), k=k, add=rng.random() < 0.5)
    if kind == "token":
        fmt, hidden = rng.choice(["q8_0", "q4_0", "q4k", "q4k"]), 256 * _log(rng, 4, 14)
        return _token(fmt, rng.choice([1, 1, 2, 3, 4, 5, 6, 8]), hidden, hidden, 128 * rng.randint(1, 8), 256 * _log(rng, 8, 74), _log(rng, 2000, 152064),
                      rng.randint(1, 8))
    if kind == "moe":
        E = rng.choice([8, 16, 60, 64])
        return dict(kind=kind, T=_log(rng, 1, 256), h=256 * rng.randint(2, 8), ff=256 * rng.randint(1, 4), E=E, top=rng.randint(1, min(8, E)))
    if kind == "experts":
        E = rng.choice([8, 60, 64, 128])
        return dict(kind=kind, T=_log(rng, 64, 4096), h=256 * rng.randint(2, 8), ff=256 * rng.randint(1, 3), E=E, top=rng.randint(1, min(8, E)))
    if kind == "decode":
        return dict(kind=kind, n=rng.randint(1, 12), layers=rng.randint(1, 6), hidden=rng.choice([1024, 2048]), heads=rng.choice([8, 16]), vocab=_log(rng, 1000, 50304),
                    E=rng.choice([8, 64]), top=rng.randint(1, 8), ff=256 * rng.randint(1, 4))
    if kind == "rows":
        return dict(kind=kind, T=_log(rng, 33, 2048), m=_log(rng, 300, 8192), k=_log(rng, 300, 4096) if rng.random() < 0.5 else 256 * rng.randint(2, 16),
                    epi=rng.choice(["relu2", "f32"]))
    kv = rng.choice([2, 4, 8, 16])
    return dict(kind="attention", T=_log(rng, 17, 2048), start=rng.choice([0, 0, rng.randint(1, 1000)]), heads=16, kv_heads=kv, hd=rng.choice([64, 128]))


# ── inputs ──

class State:
    """What a program keeps between calls; gives the library's objects back when it goes."""

    def __init__(self, **kw):
        self.graph = self.model = None
        self.__dict__.update(kw)

    def __del__(self):
        if self.graph is not None:
            self.graph.destroy()
        if self.model is not None:
            self.model.close()


_ctx = []


def _context():
    if not _ctx:
        _ctx.append(R.Context(0))
    return _ctx[0]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _normal(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda") * std


def _put_f16(w, at, v):
    w[:, at:at + 2] = v.to(torch.float16).view(torch.uint8).reshape(-1, 2)


def _weights(g, fmt, rows, k):
    """Packed blocks [rows][k / elems * bytes] whose values have a mean near zero and a spread of about 0.02."""
    elems, nbytes = BLOCK[fmt]
    n = rows * (k // elems)
    w = torch.randint(0, 256, (n, nbytes), generator=g, device="cuda", dtype=torch.uint8)
    u = torch.rand((n,), generator=g, device="cuda") + 0.5
    if fmt == "q8_0":
        w[:, 2:][w[:, 2:] == 128] = 127      # int8 values from -127
        _put_f16(w, 0, u * (0.02 / 73))
    elif fmt == "q4_0":
        _put_f16(w, 0, u * (0.02 / 4.6))
    elif fmt == "q5_0":
        _put_f16(w, 0, u * (0.02 / 9.2))
    elif fmt in ("q4k", "q5k"):              # d * scale * q - dmin * min, both 6-bit factors 31.5 on average
        mean, d = (7.5, 8e-5) if fmt == "q4k" else (15.5, 4e-5)
        _put_f16(w, 0, u * d)
        _put_f16(w, 2, u * d * mean)
    else:
        _put_f16(w, 208, u * 1.5e-5)
    return w.reshape(rows, -1)


def _token_weights(c, g):
    h, qd, kv, ff, f = c["hidden"], c["q_dim"], c["kv_dim"], c["ff"], c["fmt"]
    layers = [[_weights(g, f, m, k) for m, k in ((qd, h), (kv, h), (kv, h), (h, qd), (ff, h), (ff, h), (h, ff))] for _ in range(c["layers"])]
    return layers, _weights(g, f, c["vocab"], h)


def _decode_weights(c, g):
    L, h, q, E, ff, V = c["layers"], c["hidden"], c["heads"] * 128, c["E"], c["ff"], c["vocab"]
    w = {n: _weights(g, "q4k", r, k) for n, r, k in (("wq", L * q, h), ("wk", L * q, h), ("wv", L * q, h), ("wo", L * h, q), ("gate", L * E * ff, h),
                                                     ("up", L * E * ff, h), ("down", L * E * h, ff), ("lm_head", V, h))}
    w["tok_emb"], w["router"] = _normal(g, V, h), _normal(g, L, E, h, std=0.05)
    for n, s in (("attn_norm", (L, h)), ("ffn_norm", (L, h)), ("out_norm", (h,))):
        w[n] = 1.0 + _normal(g, *s, std=0.1)
    return w, torch.randint(0, V, (c["n"],), generator=g, device="cuda").cpu().numpy().astype(np.int32)


def _zipf(g, T, E, k):
    """Distinct experts of every token, drawn with popularity rank^-1.1, and their weights."""
    p = 1.1 * torch.log(torch.arange(1, E + 1, device="cuda", dtype=torch.float64))[torch.randperm(E, generator=g, device="cuda")]
    gumbel = -torch.log(-torch.log(torch.rand((T, E), generator=g, device="cuda", dtype=torch.float64) + 1e-12))
    idx = torch.topk(gumbel - p, k, dim=1).indices.to(torch.int32)
    w = torch.softmax(_normal(g, T, k), 1) * 0.6
    return idx.contiguous(), w.contiguous()


def _inputs(c, seed):
    """Tensors of the case, the same for prepare() and exact()."""
    g, kind = _gen(seed), c["kind"]
    if kind == "gemv":
        return dict(w=_weights(g, c["fmt"], c["m"], c["k"]), x=_normal(g, c["k"]), res=_normal(g, c["m"]) if c["add"] else None)
    if kind == "token":
        L, b = c["layers"], c["batch"]
        layers, head = _token_weights(c, g)
        return dict(layers=layers, head=head, x=_normal(g, L, b, c["hidden"]), ao=_normal(g, L, b, c["q_dim"]), x2=_normal(g, L, b, c["hidden"]),
                    res=_normal(g, L, b, c["hidden"]), bias=_normal(g, L, c["q_dim"] + 2 * c["kv_dim"], std=0.1), xh=_normal(g, b, c["hidden"]))
    if kind in ("moe", "experts"):
        E, h, ff, T = c["E"], c["h"], c["ff"], c["T"]
        d = dict(gate=_weights(g, "q4k", E * ff, h), up=_weights(g, "q4k", E * ff, h), down=_weights(g, "q4k", E * h, ff), x=_normal(g, T, h), res=_normal(g, T, h))
        if kind == "moe":
            return dict(d, router=_normal(g, E, h, std=0.02))
        idx, w = _zipf(g, T, E, c["top"])
        return dict(d, idx=idx, w=w)
    if kind == "decode":
        w, prompt = _decode_weights(c, g)
        return dict(w=w, prompt=prompt)
    if kind == "rows":
        kp = (c["k"] + 7) // 8 * 8
        w, x = torch.zeros((c["m"], kp), device="cuda", dtype=torch.bfloat16), torch.zeros((c["T"], kp), device="cuda", dtype=torch.bfloat16)
        w[:, :c["k"]] = _normal(g, c["m"], c["k"], std=c["k"] ** -0.5).bfloat16()
        x[:, :c["k"]] = _normal(g, c["T"], c["k"]).bfloat16()
        return dict(w=w, x=x)
    n, seq = c["start"] + c["T"], c["start"] + c["T"] + 32
    kc, vc = (torch.zeros((c["kv_heads"], seq, c["hd"]), device="cuda", dtype=torch.float16) for _ in range(2))
    kc[:, :n], vc[:, :n] = (_normal(g, c["kv_heads"], n, c["hd"]).half() for _ in range(2))
    return dict(q=_normal(g, c["T"], c["heads"] * c["hd"]), kc=kc, vc=vc, seq=seq)


# ── the calls ──

def _record_token(ctx, c, s):
    """One step's products; records them on ctx."""
    fmt, b = c["fmt"], c["batch"]
    h, qd, kv, ff = c["hidden"], c["q_dim"], c["kv_dim"], c["ff"]
    for l, (wq, wk, wv, wo, wg, wu, wd) in enumerate(s.layers):
        q, k, v, o, act, y = s.q[l], s.k[l], s.v[l], s.o[l], s.act[l], s.y[l]
        if b == 1:
            if fmt == "q8_0":
                bq, bk, bv = s.bias[l, :qd], s.bias[l, qd:qd + kv], s.bias[l, qd + kv:]
                R.fused_qkv_f32bias_q8_0_f32(ctx, wq, wk, wv, s.x[l], q, k, v, bq, bk, bv, qd, kv, h)
            else:
                getattr(R, "fused_qkv_%s_f32" % fmt)(ctx, wq, wk, wv, s.x[l], q, k, v, qd, kv, h)
            getattr(R, "gemv_%s_add_f32_f32in" % fmt)(ctx, wo, s.ao[l], o, s.res[l], h, qd)
            getattr(R, "fused_ffn_%s_f32" % fmt)(ctx, wg, wu, s.x2[l], act, ff, h)
            getattr(R, "gemv_%s_add_f32_f32in" % fmt)(ctx, wd, act, y, s.res[l], h, ff)
        else:
            R.gemv_batched_multi_f32(ctx, FMT[fmt], [wq, wk, wv], s.x[l], [q, k, v], [qd, kv, kv], h, b)
            R.gemv_batched_f32(ctx, FMT[fmt], wo, s.ao[l], o, s.res[l], h, qd, b)
            R.gemv_batched_multi_f32(ctx, FMT[fmt], [wg, wu], s.x2[l], [s.g, s.u], [ff, ff], h, b)
            R.silu_mul_f32(ctx, s.g, s.u, act, b * ff)
            R.gemv_batched_f32(ctx, FMT[fmt], wd, act, y, s.res[l], h, ff, b)
    if b == 1:
        getattr(R, "gemv_%s_f32in_f32out" % fmt)(ctx, s.head, s.xh, s.logits, c["vocab"], h)
    else:
        R.gemv_batched_f32(ctx, FMT[fmt], s.head, s.xh, s.logits, None, c["vocab"], h, b)


def prepare(case, seed):
    c, ctx = case, _context()
    s = State(case=c, ctx=ctx, **_inputs(c, seed))
    empty = lambda *shape, dtype=torch.float32: torch.zeros(shape, device="cuda", dtype=dtype)  # noqa: E731
    kind = c["kind"]
    if kind == "gemv":
        s.y = empty(c["m"])
    elif kind == "token":
        L, b = c["layers"], c["batch"]
        s.q, s.k, s.v = empty(L, b, c["q_dim"]), empty(L, b, c["kv_dim"]), empty(L, b, c["kv_dim"])
        s.o, s.act, s.y, s.logits = empty(L, b, c["hidden"]), empty(L, b, c["ff"]), empty(L, b, c["hidden"]), empty(b, c["vocab"])
        s.g, s.u = empty(b, c["ff"]), empty(b, c["ff"])
        torch.cuda.synchronize()
        ctx.graph_begin()
        _record_token(ctx, c, s)
        s.graph = ctx.graph_end()
    elif kind in ("moe", "experts"):
        size = R.moe_scratch_bytes if kind == "moe" else R.moe_grouped_scratch_bytes
        s.bytes = size(ctx, c["T"], c["h"], c["ff"], c["E"], c["top"])
        s.scratch, s.out = ctx.new_buffer(s.bytes), empty(c["T"], c["h"])
        if kind == "moe":
            s.idx, s.w = empty(c["T"], c["top"], dtype=torch.int32), empty(c["T"], c["top"])
    elif kind == "decode":
        cfg = R.ModelCfg(n_layers=c["layers"], hidden=c["hidden"], n_heads=c["heads"], n_kv_heads=c["heads"], head_dim=128, vocab=c["vocab"], n_experts=c["E"],
                         top_k=c["top"], ff=c["ff"], max_seq=2048, renorm=0, eps=1e-5, theta=10000.0)
        torch.cuda.synchronize()
        s.model = R.Model(ctx, cfg, s.w)
    elif kind == "rows":
        s.y = empty(c["T"], (c["m"] + 7) // 8 * 8, dtype=torch.float32 if c["epi"] == "f32" else torch.bfloat16)
    else:
        s.out = empty(c["T"], c["heads"] * c["hd"], dtype=torch.bfloat16)
    torch.cuda.synchronize()
    return s


def run(state):
    s, c, ctx = state, state.case, state.ctx
    kind = c["kind"]
    if kind == "gemv":
        if c["add"]:
            getattr(R, "gemv_%s_add_f32_f32in" % c["fmt"])(ctx, s.w, s.x, s.y, s.res, c["m"], c["k"])
        else:
            getattr(R, "gemv_%s_f32in_f32out" % c["fmt"])(ctx, s.w, s.x, s.y, c["m"], c["k"])
        return s.y
    if kind == "token":
        s.graph.launch()
        return [s.q, s.k, s.v, s.o, s.act, s.y, s.logits]
    if kind == "moe":
        R.moe_layer_q4k(ctx, s.router, s.gate, s.up, s.down, s.x, s.res, s.out, s.idx, s.w, s.scratch, s.bytes, c["T"], c["h"], c["ff"], c["E"], c["top"], 0)
        return [s.out, s.w]
    if kind == "experts":
        R.moe_experts_grouped_q4k_bf16(ctx, s.gate, s.up, s.down, s.x, s.idx, s.w, s.res, s.out, s.scratch, s.bytes, c["T"], c["h"], c["ff"], c["E"], c["top"])
        return s.out
    if kind == "decode":
        s.model.generate_greedy(s.prompt, 0)
        return s.model.logits()
    if kind == "rows":
        R.gemm_bf16_rows(ctx, s.w, s.x, s.y, s.y.shape[1], c["T"], c["m"], c["k"], 0, R.EPI_F32 if c["epi"] == "f32" else R.EPI_RELU2, None, None)
        return s.y[:, :c["m"]]
    R.prefill_attention_f16kv(ctx, s.q, s.kc, s.vc, s.out, c["T"], c["heads"], c["kv_heads"], c["hd"], s.seq, c["start"])
    return s.out


# ── what a pass cannot do without ──

def _packed(fmt, m, k):
    return m * (k // BLOCK[fmt][0]) * BLOCK[fmt][1]


def work(case):
    c, kind = case, case["kind"]
    if kind == "gemv":
        return dict(bytes=_packed(c["fmt"], c["m"], c["k"]) + 4 * (c["k"] + c["m"] * (2 if c["add"] else 1)), flops=2 * c["m"] * c["k"])
    if kind == "token":
        h, qd, kv, ff, b, f = c["hidden"], c["q_dim"], c["kv_dim"], c["ff"], c["batch"], c["fmt"]
        mats = [(qd, h), (kv, h), (kv, h), (h, qd), (ff, h), (ff, h), (h, ff)]
        w = c["layers"] * sum(_packed(f, m, k) for m, k in mats) + _packed(f, c["vocab"], h)
        v = c["layers"] * (3 * h + 2 * qd + 2 * kv + ff + 2 * h) + h + c["vocab"]      # inputs, residuals and outputs
        return dict(bytes=w + 4 * b * v, flops=2 * b * (c["layers"] * sum(m * k for m, k in mats) + c["vocab"] * h))
    if kind in ("moe", "experts"):
        T, h, ff, E, top = c["T"], c["h"], c["ff"], c["E"], c["top"]
        used = E * (1 - (1 - top / E) ** T)                                            # experts that some token picks
        per = 2 * _packed("q4k", ff, h) + _packed("q4k", h, ff)
        return dict(bytes=used * per + 12 * T * h + 8 * T * top + (4 * E * h if kind == "moe" else 0), flops=T * top * 6 * h * ff + (2 * T * E * h if kind == "moe" else 0))
    if kind == "decode":
        h, q, ff = c["hidden"], c["heads"] * 128, c["ff"]
        layer = 3 * _packed("q4k", q, h) + _packed("q4k", h, q) + c["top"] * (2 * _packed("q4k", ff, h) + _packed("q4k", h, ff)) + 4 * c["E"] * h
        return dict(bytes=c["n"] * c["layers"] * layer + _packed("q4k", c["vocab"], h) + 4 * c["vocab"],
                    flops=2 * c["n"] * c["layers"] * (4 * q * h + 3 * c["top"] * ff * h) + 2 * c["vocab"] * h)
    if kind == "rows":
        return dict(bytes=2 * (c["m"] + c["T"]) * c["k"] + c["T"] * c["m"] * (4 if c["epi"] == "f32" else 2), flops=2 * c["T"] * c["m"] * c["k"])
    T, n, hd = c["T"], c["start"] + c["T"], c["hd"]
    return dict(bytes=T * c["heads"] * hd * 6 + 4 * c["kv_heads"] * n * hd, flops=4 * c["heads"] * hd * (T * c["start"] + T * (T + 1) // 2))


def tolerance(case):
    kind = case["kind"]
    if kind in ("gemv", "token"):
        # activations meet the 4-bit and 8-bit weights as 16-bit integers with a scale per block
        return {"rel": 1e-5} if case["fmt"] in ("q5_0", "q5k", "q6k") else {"rel": 3e-4}
    if kind == "moe":
        return {"rel": 3e-4}
    if kind == "experts":
        return {"rel": 5e-3}      # bf16 weights, activations and products of gate and up
    if kind == "decode":
        return {"rel": 1e-2}      # f16 cache; a near tie among the experts can fall on the other side
    if kind == "rows":
        return {"rel": 1e-5} if case["epi"] == "f32" else {"rel": 1e-2}
    return {"rel": 1e-2}


# ── the same in 64 bits ──

def _f16(w, at):
    return w[:, at:at + 2].contiguous().view(torch.float16).double()


def _scales(s):
    """6-bit scales and minimums [n][8] of 12 packed bytes."""
    lo, hi = s[:, 0:4], s[:, 4:8]
    last = s[:, 8:12]
    sc = torch.cat([lo & 63, (last & 15) | ((lo >> 6) << 4)], 1)
    mn = torch.cat([hi & 63, (last >> 4) | ((hi >> 6) << 4)], 1)
    return sc, mn


def _values(fmt, w, k):
    """Weights [rows][k] in 64 bits of packed rows."""
    rows = w.shape[0]
    w = w.reshape(-1, BLOCK[fmt][1])
    n = w.shape[0]
    if fmt == "q8_0":
        return (_f16(w, 0) * w[:, 2:].contiguous().view(torch.int8).double()).reshape(rows, k)
    if fmt == "q4_0":
        q = torch.stack([w[:, 2:] & 15, w[:, 2:] >> 4], 2).reshape(n, 32)      # neighbours share a byte
        return (_f16(w, 0) * (q.double() - 8)).reshape(rows, k)
    bits = torch.arange(8, device=w.device, dtype=torch.uint8)
    if fmt == "q5_0":
        fifth = ((w[:, 2:6, None] >> bits) & 1).reshape(n, 32)
        q = torch.cat([w[:, 6:] & 15, w[:, 6:] >> 4], 1) | (fifth << 4)
        return (_f16(w, 0) * (q.double() - 16)).reshape(rows, k)
    if fmt == "q6k":
        ql, qh, sc = w[:, :128].reshape(n, 2, 2, 32), w[:, 128:192].reshape(n, 2, 32), w[:, 192:208].contiguous().view(torch.int8).reshape(n, 2, 8)
        parts = []
        for i in range(4):
            low = (ql[:, :, i % 2] & 15) if i < 2 else (ql[:, :, i % 2] >> 4)
            q = (low | (((qh >> (2 * i)) & 3) << 4)).double() - 32
            parts.append(q * sc[:, :, 2 * i, None].double())                   # the first of a group's two scales serves all 32
        return (_f16(w, 208)[:, :, None, None] * torch.stack(parts, 2)).reshape(rows, k)
    sc, mn = _scales(w[:, 4:16])
    qs = w[:, 16:] if fmt == "q4k" else w[:, 48:]
    q = torch.stack([qs.reshape(n, 4, 32) & 15, qs.reshape(n, 4, 32) >> 4], 2)  # [n][chunk][half][32]
    if fmt == "q5k":
        q = q | (((w[:, 16:48, None] >> bits) & 1).reshape(n, 4, 2, 32) << 4)
    sc, mn = (t.reshape(n, 2, 4).transpose(1, 2)[..., None].double() for t in (sc, mn))
    d, dmin = _f16(w, 0)[..., None, None], _f16(w, 2)[..., None, None]
    return (d * sc * q.double() - dmin * mn).reshape(rows, k)


def _times(fmt, w, x, step=16384):
    """x [b][k] times the packed matrix: [b][rows]."""
    k = x.shape[-1]
    return torch.cat([x @ _values(fmt, w[i:i + step], k).T for i in range(0, w.shape[0], step)], -1)


def _silu(v):
    return v * torch.sigmoid(v)


def _experts(d, c, x, idx, w):
    """Weighted sum of the chosen experts' outputs for x [T][h]."""
    E, h, ff = c["E"], x.shape[1], c["ff"]
    gate, up, down = d["gate"].reshape(E, ff, -1), d["up"].reshape(E, ff, -1), d["down"].reshape(E, h, -1)
    out = torch.zeros_like(x)
    for e in range(E):
        t, i = torch.nonzero(idx == e, as_tuple=True)
        if t.numel():
            act = _silu(_times("q4k", gate[e], x[t])) * _times("q4k", up[e], x[t])
            out.index_add_(0, t, w[t, i, None] * _times("q4k", down[e], act))
    return out


def _route(router, x, top):
    p = torch.softmax(x @ router.double().T, -1)
    w, idx = torch.topk(p, top, dim=-1)
    return idx, w


def _norm(x, gain):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gain.double()


def _exact_decode(c, d):
    L, h, H, E, ff = c["layers"], c["hidden"], c["heads"], c["E"], c["ff"]
    w, n = d["w"], c["n"]
    x = w["tok_emb"][torch.from_numpy(d["prompt"]).long().cuda()].double()
    freq = 10000.0 ** (-torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)
    angle = torch.arange(n, device="cuda", dtype=torch.float64)[:, None, None] * freq
    hide = torch.triu(torch.full((n, n), -math.inf, device="cuda", dtype=torch.float64), 1)

    def turned(v):
        a, b = v[..., :64], v[..., 64:]
        return torch.cat([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()], -1)
    for l in range(L):
        of = lambda name, rows: w[name][l * rows:(l + 1) * rows]  # noqa: E731
        y = _norm(x, w["attn_norm"][l])
        q, k, v = (_times("q4k", of(name, H * 128), y).reshape(n, H, 128) for name in ("wq", "wk", "wv"))
        p = torch.softmax(torch.einsum("ihd,jhd->hij", turned(q), turned(k)) / math.sqrt(128) + hide, -1)
        x = x + _times("q4k", of("wo", h), torch.einsum("hij,jhd->ihd", p, v).reshape(n, -1))
        y = _norm(x, w["ffn_norm"][l])
        idx, p = _route(w["router"][l], y, c["top"])
        x = x + _experts(dict(gate=of("gate", E * ff), up=of("up", E * ff), down=of("down", E * h)), c, y, idx, p)
    return _times("q4k", w["lm_head"], _norm(x[-1:], w["out_norm"]))[0].cpu().numpy()


def exact(case, seed):
    c, kind = case, case["kind"]
    d = _inputs(c, seed)
    if kind == "gemv":
        y = _times(c["fmt"], d["w"], d["x"].double()[None])[0]
        return y + d["res"].double() if c["add"] else y
    if kind == "token":
        f, out = c["fmt"], [[] for _ in range(6)]
        bias = torch.split(d["bias"].double(), [c["q_dim"], c["kv_dim"], c["kv_dim"]], 1)
        for l, (wq, wk, wv, wo, wg, wu, wd) in enumerate(d["layers"]):
            x, x2, res = d["x"][l].double(), d["x2"][l].double(), d["res"][l].double()
            for j, m in enumerate((wq, wk, wv)):
                out[j].append(_times(f, m, x) + (bias[j][l] if f == "q8_0" and c["batch"] == 1 else 0))
            out[3].append(_times(f, wo, d["ao"][l].double()) + res)
            out[4].append(_silu(_times(f, wg, x2)) * _times(f, wu, x2))
            out[5].append(_times(f, wd, out[4][-1]) + res)
        return [torch.stack(o) for o in out] + [_times(f, d["head"], d["xh"].double())]
    if kind == "moe":
        x = d["x"].double()
        idx, w = _route(d["router"], x, c["top"])
        return [_experts(d, c, x, idx, w) + d["res"].double(), w]
    if kind == "experts":
        return _experts(d, c, d["x"].double(), d["idx"].long(), d["w"].double()) + d["res"].double()
    if kind == "decode":
        return _exact_decode(c, d)
    if kind == "rows":
        y = d["x"].double() @ d["w"].double().T
        return y if c["epi"] == "f32" else torch.relu(y) ** 2
    T, H, G, hd, n = c["T"], c["heads"], c["kv_heads"], c["hd"], c["start"] + c["T"]
    q = d["q"].double().reshape(T, H, hd)
    hide = torch.triu(torch.full((T, n), -math.inf, device="cuda", dtype=torch.float64), c["start"] + 1)
    out = torch.empty((T, H, hd), device="cuda", dtype=torch.float64)
    for i in range(H):
        j = i // (H // G)
        p = torch.softmax(q[:, i] @ d["kc"][j, :n].double().T / math.sqrt(hd) + hide, -1)
        out[:, i] = p @ d["vc"][j, :n].double()
    return out.reshape(T, H * hd)
