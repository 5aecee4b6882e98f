"""GPU parity tests of the batched prefill (crates/engine/src/prefill.rs:29-255) through the C ABI.

The device path rounds GEMM operands to bf16 and attention operands to f16; oracle/prefill.py restates exactly that
arithmetic (f64 accumulation).  Single kernels are held to it at 1e-3 of the output scale (5e-3 for the bf16-rounded
attention output: one bf16 ulp is 2^-8 of the value), the whole pass over several tokens at 5e-3 rms (see the test).  Against the f32 decode oracle, which the reference's formulas pin, the same
quantities agree to bf16 operand rounding; tests/test_oracle.py holds that comparison."""
import numpy as np
import pytest

from helpers import assert_close

pytestmark = pytest.mark.gpu


def bf16_bits_to_f32(u16):
    return (u16.astype(np.uint32) << 16).view(np.float32)


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("T,start", [(1, 0), (63, 0), (64, 0), (65, 0), (200, 0), (70, 37)])
def test_causal_attention_kernel(ctx, oracle, hd, T, start):
    import runit_mac_b200 as R
    from oracle import prefill as OP
    heads, kvh, max_seq = 4, 2, 320
    rng = np.random.default_rng(T * 7 + hd + start)
    q = rng.normal(0, 1, (T, heads * hd)).astype(np.float32)
    kc = np.zeros((kvh, max_seq, hd), np.float16)
    vc = np.zeros((kvh, max_seq, hd), np.float16)
    kc[:, :start + T] = rng.normal(0, 1, (kvh, start + T, hd)).astype(np.float16)
    vc[:, :start + T] = rng.normal(0, 1, (kvh, start + T, hd)).astype(np.float16)
    kc[:, start + T:] = np.float16(1e4)        # rows past the data must never contribute
    vc[:, start + T:] = np.float16(1e4)
    ob = ctx.new_buffer(T * heads * hd * 2)
    R.prefill_attention_f16kv(ctx, ctx.buffer_from(q), ctx.buffer_from(kc), ctx.buffer_from(vc), ob, T, heads, kvh, hd, max_seq, start)
    ctx.flush()
    got = bf16_bits_to_f32(ob.download(np.uint16, T * heads * hd)).reshape(T, heads * hd)
    ref = OP.causal_attention_f16(q, kc, vc, heads, kvh, hd, start_pos=start)
    assert_close(oracle, ref, got, rel_tol=5e-3, what="prefill attention hd=%d T=%d start=%d" % (hd, T, start))


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("T,start,heads,kvh", [(65, 63, 2, 2), (127, 1, 4, 1), (128, 0, 2, 1), (129, 127, 2, 2), (257, 300, 6, 3)])
def test_causal_attention_tensor_core_tiles(ctx, oracle, hd, T, start, heads, kvh):
    """Edges of the 128-query tiles and 128-key blocks; NaN in the cache behind the data must not show; a large score decides its
    row.  Bound: q is rounded alike on both sides; P is rounded to f16 relative to the maximum over blocks of other lengths than the
    restatement's, so either side's weights are off by 2^-11, which is d = 2 * 2^-11 * (P . |V|) of an output (f32 sums are far
    below), and the output's rounding to bf16 is half an ulp, 2^-8 of it."""
    import runit_mac_b200 as R
    from oracle import prefill as OP
    n, max_seq = start + T, start + T + 40
    rng = np.random.default_rng(T * 11 + hd + start)
    q = rng.normal(0, 1, (T, heads * hd)).astype(np.float32)
    q[T // 2] *= 12.0
    kc = np.full((kvh, max_seq, hd), np.nan, np.float16)
    vc = np.full((kvh, max_seq, hd), np.nan, np.float16)
    kc[:, :n] = rng.normal(0, 1, (kvh, n, hd)).astype(np.float16)
    vc[:, :n] = rng.normal(0, 1, (kvh, n, hd)).astype(np.float16)
    ob = ctx.new_buffer(T * heads * hd * 2)
    R.prefill_attention_f16kv(ctx, ctx.buffer_from(q), ctx.buffer_from(kc), ctx.buffer_from(vc), ob, T, heads, kvh, hd, max_seq, start)
    ctx.flush()
    got = bf16_bits_to_f32(ob.download(np.uint16, T * heads * hd)).reshape(T, heads * hd)
    kc[:, n:], vc[:, n:] = 0, 0
    ref = OP.causal_attention_f16(q, kc, vc, heads, kvh, hd, start_pos=start)
    d = 2.0 ** -10 * OP.causal_attention_f16(q, kc, np.abs(vc), heads, kvh, hd, start_pos=start) + 1e-6
    assert np.isfinite(got).all()
    worst = (np.abs(got - ref) / (d + 2.0 ** -8 * (np.abs(ref) + d))).max()
    assert worst <= 1.0, worst


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("T,start", [(1, 127), (1, 128), (2, 254), (129, 128), (3, 509), (256, 129), (1, 640)])
def test_causal_attention_chains_of_even_and_odd_blocks(ctx, oracle, hd, T, start):
    """One to six blocks of keys: a chain without a block, chains of one and of several, a last block with a single visible key.  Same bound."""
    test_causal_attention_tensor_core_tiles(ctx, oracle, hd, T, start, 2, 1)


def test_causal_attention_weights_are_relative_to_the_maximum(ctx, oracle):
    """Two keys of the second block decide the row, 5.3 bits above the first block's largest score, and their values cancel to a few
    thousandths: what is left shows how their weights were rounded to f16.  Relative to the row maximum the largest is 1 and exact, as in the
    restatement, and the outputs agree to the rounding to bf16; relative to another reference both weights are off by up to 2^-12, which
    would be 2e-4 here."""
    import runit_mac_b200 as R
    from oracle import prefill as OP
    hd, n = 64, 256
    q = np.zeros((1, hd), np.float32)
    q[0, 0] = 8.0                                   # score = the first element of the key
    kc, vc = np.zeros((1, n, hd), np.float16), np.zeros((1, n, hd), np.float16)
    kc[0, :, 0] = -14
    kc[0, 5, 0], kc[0, 200, 0], kc[0, 201, 0] = 0, 3.7, 2.8
    vc[0, 200] = 1
    vc[0, 201] = -np.exp(0.9) * (1 + np.linspace(-0.004, 0.004, hd))
    ob = ctx.new_buffer(hd * 2)
    R.prefill_attention_f16kv(ctx, ctx.buffer_from(q), ctx.buffer_from(kc), ctx.buffer_from(vc), ob, 1, 1, 1, hd, n, n - 1)
    ctx.flush()
    got = bf16_bits_to_f32(ob.download(np.uint16, hd))
    ref = OP.causal_attention_f16(q, kc, vc, 1, 1, hd, start_pos=n - 1).reshape(-1)
    assert np.abs(ref).max() < 0.01
    assert (np.abs(got - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-6).all(), np.abs(got - ref).max()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("T,start,key", [(200, 0, 70), (200, 37, 101), (127, 1, 127), (300, 100, 256), (40, 300, 339)])
def test_causal_attention_hidden_value_does_not_show(ctx, oracle, hd, T, start, key, bad):
    """One value of one position is not finite: the queries before that position do not see it, the others see it in its dimension
    and nowhere else.  What stays finite is held to the bound of the kernel's other tests, against a cache with a 0 in its place."""
    import runit_mac_b200 as R
    from oracle import prefill as OP
    heads, kvh, n, d = 4, 2, start + T, hd - 3
    rng = np.random.default_rng(T + hd + key)
    q = rng.normal(0, 1, (T, heads * hd)).astype(np.float32)
    kc, vc = (rng.normal(0, 1, (kvh, n, hd)).astype(np.float16) for _ in range(2))
    vc[1, key, d] = bad
    ob = ctx.new_buffer(T * heads * hd * 2)
    R.prefill_attention_f16kv(ctx, ctx.buffer_from(q), ctx.buffer_from(kc), ctx.buffer_from(vc), ob, T, heads, kvh, hd, n, start)
    ctx.flush()
    got = bf16_bits_to_f32(ob.download(np.uint16, T * heads * hd)).reshape(T, heads, hd)
    vc[1, key, d] = 0
    ref = OP.causal_attention_f16(q, kc, vc, heads, kvh, hd, start_pos=start).reshape(T, heads, hd)
    sees = np.zeros(got.shape, bool)
    sees[max(key - start, 0):, 2:, d] = True
    assert not np.isfinite(got[sees]).any()
    assert_close(oracle, ref[~sees], got[~sees], rel_tol=5e-3, what="value of position %d" % key)


@pytest.mark.parametrize("hd", [128, 64])
def test_causal_attention_calls_in_a_row(ctx, hd):
    """Calls that follow one another without a wait, each with more blocks than SMs: a dependent call starts while the one before
    it still holds tensor memory.  Every call gives the same bits."""
    import runit_mac_b200 as R
    T, heads = 1300, 16
    rng = np.random.default_rng(hd)
    q = ctx.buffer_from(rng.normal(0, 1, (T, heads * hd)).astype(np.float32))
    kc, vc = (ctx.buffer_from(rng.normal(0, 1, (heads, T, hd)).astype(np.float16)) for _ in range(2))
    outs = [ctx.new_buffer(T * heads * hd * 2) for _ in range(6)]
    for ob in outs:
        R.prefill_attention_f16kv(ctx, q, kc, vc, ob, T, heads, heads, hd, T, 0)
    ctx.flush()
    first = outs[0].download(np.uint16, T * heads * hd)
    assert np.isfinite(bf16_bits_to_f32(first)).all()
    for ob in outs[1:]:
        assert np.array_equal(ob.download(np.uint16, T * heads * hd), first)


def test_small_model_prefill_matches_restatement_and_decode(ctx, oracle):
    import runit_mac_b200 as R
    from oracle import prefill as OP
    from test_decode_gpu import SMALL, build_model
    O = oracle
    model, ocfg, ow, host = build_model(ctx, R, O, SMALL, 11, device_fill=False, zero_mean=True)
    hostw = {k: v for k, v in host.items() if not k.startswith("_")}
    for n in (1, 5, 40, 57):
        prompt = np.random.default_rng(n).integers(0, SMALL["vocab"], n).astype(np.int32)
        tok = model.prefill(prompt)
        logits = model.logits()
        rtok, rlogits, kc, vc = OP.prefill(SMALL, hostw, prompt)
        spread = float(np.std(rlogits))
        if n == 1:
            # one token: attention is the value row itself, every GEMM and the MoE block are compared at the kernel bar
            assert_close(O, rlogits, logits, rel_tol=1e-3, what="prefill logits, 1 token")
        else:
            # several stages in a row: where the device's f32 sum and the restatement's f64 sum fall on different sides of a
            # bf16 (or f16) rounding boundary the operand of the next stage differs by one ulp (2^-8 of its value); a few
            # per cent of the operands do, which adds about 6e-4 rms per stage.  Held to 5e-3 rms / 2e-2 at worst.
            d = np.abs(logits - rlogits)
            assert np.sqrt((d ** 2).mean()) <= 5e-3 * spread and d.max() <= 2e-2 * spread, (n, d.max(), np.sqrt((d ** 2).mean()), spread)
        assert tok == rtok or abs(rlogits[tok] - rlogits[rtok]) <= 2e-2 * spread
        # decoding continues from the cache the prefill filled: the next steps agree with the decode oracle run on the
        # restatement's cache (f16 rounding of k and v can differ in the last bit where bf16 sums differ: logits at 1e-2)
        out = model.generate_greedy(np.array([tok], np.int32), 4, start_pos=n)
        kc = kc.copy(); vc = vc.copy()
        t = tok
        for step in range(3):
            t_ref, l_ref = O.decode_step(ocfg, ow, kc, vc, int(t), n + step, want_logits=True)
            if step == 0:
                model.generate_greedy(np.array([tok], np.int32), 0, start_pos=n)      # one step: logits of position n
                d = np.abs(model.logits() - l_ref)
                assert d.max() <= 2e-2 * float(np.std(l_ref)), (n, d.max(), float(np.std(l_ref)))
            t = t_ref
        # against the decoder run token by token on the device (f32 path): same next token unless the logits are that close
        model2 = R.Model(ctx, host["_cfg"], host["_dev"])
        o2 = model2.generate_greedy(prompt, 1, skip_prompt_logits=False)
        if o2[n - 1] != tok:
            assert abs(rlogits[tok] - rlogits[o2[n - 1]]) <= 8e-2 * spread
        model2.close()
        assert out[0] >= 0
    with pytest.raises(R.KernelError):
        model.prefill(np.array([SMALL["vocab"]], np.int32))                  # InvalidTokenId, prefill.rs:55-57
    with pytest.raises(R.KernelError):
        model.prefill(np.zeros(SMALL["max_seq"] + 1, np.int32))
    model.close()


def test_olmoe_shaped_prefill_128_tokens(ctx, oracle):
    """The 128-token prompt of the decode benchmark through the batched pass at the full OLMoE shape: the logits of the
    last position against the f32 decode oracle fed token by token (bf16 operand rounding: 1e-2 of the spread rms)."""
    import runit_mac_b200 as R
    from test_decode_gpu import OLMOE_EMB_SIGMA, OLMOE_WEIGHT_SIGMA, build_model
    O = oracle
    cfg = dict(n_layers=16, hidden=2048, n_heads=16, n_kv_heads=16, head_dim=128, vocab=50304, n_experts=64, top_k=8, ff=1024,
               max_seq=2048, renorm=0, eps=1e-5, theta=10000.0)
    model, ocfg, ow, host = build_model(ctx, R, O, cfg, 1004, device_fill=True, zero_mean=True, weight_sigma=OLMOE_WEIGHT_SIGMA,
                                        emb_sigma=OLMOE_EMB_SIGMA)
    prompt = np.random.default_rng(1004).integers(0, 50304, 128).astype(np.int32)
    tok = model.prefill(prompt)
    logits = model.logits()
    L, kvh, S, hd = 16, 16, 2048, 128
    kc = np.zeros((L, kvh, S, hd), np.float16)
    vc = np.zeros_like(kc)
    for pos, t in enumerate(prompt[:-1]):
        O.decode_step(ocfg, ow, kc, vc, int(t), pos)
    ref_tok, ref_logits = O.decode_step(ocfg, ow, kc, vc, int(prompt[-1]), len(prompt) - 1, want_logits=True)
    spread = float(np.std(ref_logits))
    d = np.abs(logits - ref_logits)
    assert np.sqrt((d ** 2).mean()) <= 1e-2 * spread and d.max() <= 8e-2 * spread, (d.max(), np.sqrt((d ** 2).mean()), spread)
    assert tok == ref_tok or abs(ref_logits[tok] - ref_logits[ref_tok]) <= 8e-2 * spread
    # and the decoder continues from that cache
    out = model.generate_greedy(np.array([tok], np.int32), 8, start_pos=128)
    assert (out >= 0).all()
    model.close()


@pytest.mark.parametrize("T", [1, 100, 300])
def test_dense_ffn_block(ctx, oracle, T):
    """The dense feed-forward block of a prefill pass (prefill.rs:217-227) on the tensor cores, with and without the RMSNorm in
    front and the residual, against the bf16-operand restatement (the batched block's oracle with one expert, weight 1)."""
    import runit_mac_b200 as R
    O = oracle
    h, ff = 512, 768
    rng = np.random.default_rng(40 + T)
    wg, wu, wd = O.rand_q4k(rng, ff, h), O.rand_q4k(rng, ff, h), O.rand_q4k(rng, h, ff)
    x = rng.normal(0, 1, (T, h)).astype(np.float32)
    res = rng.normal(0, 1, (T, h)).astype(np.float32)
    gamma = rng.normal(1, 0.1, h).astype(np.float32)
    nb = ctx.lib.runit_ffn_q4k_bf16_scratch_bytes(T, h, ff)
    scratch = ctx.new_buffer(nb)
    wb = [ctx.buffer_from(w) for w in (wg, wu, wd)]
    ob = ctx.new_buffer(T * h * 4)
    routing = (np.zeros((T, 1), np.int32), np.ones((T, 1), np.float32))
    for use_gamma, use_res in ((False, False), (True, True), (False, True)):
        xin = O.rms_norm_f32(x, gamma, 1e-5) if use_gamma else x
        ref, _, _ = O.moe_grouped_q4k_bf16(None, wg, wu, wd, xin, h=h, ff=ff, E=1, top_k=1, residual=res if use_res else None, routing=routing)
        R.ffn_q4k_bf16(ctx, *wb, ctx.buffer_from(x), ctx.buffer_from(gamma) if use_gamma else None, 1e-5,
                       ctx.buffer_from(res) if use_res else None, ob, scratch, nb, T, h, ff)
        ctx.flush()
        got = ob.download(np.float32, T * h).reshape(T, h)
        scale = np.maximum(np.abs(ref), np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
        rel = float((np.abs(got - ref) / scale).max())
        assert rel <= 4e-3, (T, use_gamma, use_res, rel)


def test_dense_ffn_block_of_many_tokens(ctx, oracle):
    """Several items per pair of CTAs, a last token tile of 139; nothing behind the last token is written."""
    import torch
    import runit_mac_b200 as R
    from test_moe_grouped_gpu import expert_outputs, values
    O = oracle
    T, h, ff = 19851, 512, 768
    rng = np.random.default_rng(4)
    ws = [O.rand_q4k(rng, r, c) for r, c in ((ff, h), (ff, h), (h, ff))]
    x = torch.from_numpy(rng.normal(0, 1, (T, h)).astype(np.float32)).cuda()
    nb = ctx.lib.runit_ffn_q4k_bf16_scratch_bytes(T, h, ff)
    scratch, out = ctx.new_buffer(nb), torch.full((T + 64, h), 7.5, device="cuda")
    torch.cuda.synchronize()
    wb = [ctx.buffer_from(w) for w in ws]
    R.ffn_q4k_bf16(ctx, *wb, x, None, 1e-5, None, out, scratch, nb, T, h, ff)
    ctx.flush()
    assert (out[T:] == 7.5).all()
    ref = expert_outputs(x, *(values(O, w, 1, r, c)[0] for w, r, c in zip(ws, (ff, ff, h), (h, h, ff))))
    scale = torch.maximum(ref.abs(), (ref * ref).mean().sqrt())
    assert ((out[:T].double() - ref).abs() / scale).max() <= 4e-3        # the bound of the block of few tokens: one bf16 rounding of an activation
