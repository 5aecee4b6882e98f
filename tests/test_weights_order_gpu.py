"""Weights that the kernel directly before a GEMV writes: ops of a context are in order on its stream, the caller's own kernels on an
adopted stream and the library's fills included, although a dependent launch requests its first weights early elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tag,m,k,block,at", [("q8_0", 896, 896, 34, (0,)), ("q8_0", 4864, 896, 34, (0,)), ("q6k", 2048, 2048, 210, (208,)), ("q6k", 100, 256, 210, (208,)),
                                              ("q6k", 8192, 768, 210, (208,)), ("q6k", 8199, 512, 210, (208,)),
                                              ("q5k", 3584, 1792, 176, (0, 2))])
def test_callers_kernel_on_an_adopted_stream(tag, m, k, block, at):
    import torch
    import runit_mac_b200 as R
    stream = torch.cuda.Stream()
    ctx = R.Context(0, stream=stream.cuda_stream)
    op = getattr(R, "gemv_%s_f32in_f32out" % tag)
    try:
        with torch.cuda.stream(stream):
            n = m * k // (32 if block == 34 else 256)
            g = torch.Generator(device="cuda").manual_seed(m)
            sets = torch.randint(0, 256, (2, n, block), generator=g, device="cuda", dtype=torch.uint8)
            scale = (torch.rand((2, n, 1), generator=g, device="cuda") + 0.5).half().view(torch.uint8)
            for a in at:
                sets[:, :, a:a + 2] = scale
            w, x = torch.zeros_like(sets[0]), torch.randn(k, generator=g, device="cuda")
            y = torch.zeros(50, m, device="cuda")
            ref = torch.zeros(2, m, device="cuda")
            for i in range(2):
                torch.bitwise_xor(sets[i], 0, out=w)
                torch.cuda.synchronize()
                op(ctx, w, x, ref[i], m, k)
                ctx.flush()
            for i in range(50):
                torch.bitwise_xor(sets[i % 2], 0, out=w)          # a kernel, not a copy
                op(ctx, w, x, y[i], m, k)
            ctx.flush()
            assert torch.isfinite(ref).all() and not torch.equal(ref[0], ref[1])
            for i in range(50):
                assert torch.equal(y[i], ref[i % 2]), i
    finally:
        ctx.close()


@pytest.mark.parametrize("rows,k,batch", [((896,), 1024, 2), ((4864, 300, 128), 768, 7)])
def test_callers_kernel_before_a_batched_gemv(rows, k, batch):
    """One matrix, or three in one launch."""
    import torch
    import runit_mac_b200 as R
    stream = torch.cuda.Stream()
    ctx = R.Context(0, stream=stream.cuda_stream)
    ctx.set_tuning("gemv_tc", 1)
    try:
        with torch.cuda.stream(stream):
            g = torch.Generator(device="cuda").manual_seed(k)
            sets = [torch.randint(0, 256, (2, m * k // 32, 34), generator=g, device="cuda", dtype=torch.uint8) for m in rows]
            for s in sets:
                s[:, :, :2] = (torch.rand(s.shape[:2] + (1,), generator=g, device="cuda") + 0.5).half().view(torch.uint8)
            ws, x = [torch.zeros_like(s[0]) for s in sets], torch.randn(batch, k, generator=g, device="cuda")
            ys = [torch.zeros(52, batch, m, device="cuda") for m in rows]

            def call(i, which):
                for s, w in zip(sets, ws):
                    torch.bitwise_xor(s[which], 0, out=w)             # a kernel, not a copy
                if i < 2:
                    torch.cuda.synchronize()
                if len(rows) == 1:
                    R.gemv_batched_f32(ctx, 0, ws[0], x, ys[0][i], None, rows[0], k, batch)
                else:
                    R.gemv_batched_multi_f32(ctx, 0, ws, x, [y[i] for y in ys], rows, k, batch)
                if i < 2:
                    ctx.flush()
            for i in range(52):
                call(i, i % 2)
            ctx.flush()
            for y in ys:
                assert torch.isfinite(y).all() and not torch.equal(y[0], y[1])
                for i in range(2, 52):
                    assert torch.equal(y[i], y[i % 2]), i
    finally:
        ctx.close()


@pytest.mark.parametrize("batch", [1, 4])
def test_fill_before_a_gemv(ctx, batch):
    import runit_mac_b200 as R
    m, k = 896, 896 if batch == 1 else 1024
    w, x = ctx.new_buffer(m * k // 32 * 34), ctx.buffer_from(np.random.default_rng(0).normal(0, 1, batch * k).astype(np.float32))
    outs = []
    ctx.set_tuning("gemv_tc", 1)
    for wait in (True, False):
        ys = [ctx.new_buffer(batch * m * 4) for _ in range(20)]
        for i, y in enumerate(ys):
            R.fill_weights(ctx, R.FMT_Q8_0, w, m * k // 32, i % 3, 0.02)
            if wait:
                ctx.flush()
            if batch == 1:
                R.gemv_q8_0_f32in_f32out(ctx, w, x, y, m, k)
            else:
                R.gemv_batched_f32(ctx, R.FMT_Q8_0, w, x, y, None, m, k, batch)
        ctx.flush()
        outs.append([y.download(np.float32, batch * m) for y in ys])
    ctx.set_tuning("gemv_tc", 0)
    assert not np.array_equal(outs[0][0], outs[0][1])
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
