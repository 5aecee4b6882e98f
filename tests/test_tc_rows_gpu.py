"""Packed rows times a few columns on tcgen05 (tc_rows.cuh): the batched Q8_0 GEMV and the MoE layer with its slots sorted by expert, at the edges of their
tiles and rings.

Bound: an activation keeps 24 bits (Q4_K, and Q6_K from K = 2048 on, 22: two f16 halves of x / 2^e, error <= 2^-22 of it or 2^-35 of the largest of its 256), products are exact, sums
are f32: 2^-24 of the running sum per addition along 32 products, 8 blocks and K / 256 units.  2e-5 of max(|ref|, rms) holds with room."""
import numpy as np
import pytest

from helpers import assert_close
from test_moe_slots_gpu import run

pytestmark = pytest.mark.gpu


@pytest.fixture
def on_tc(ctx):
    """Small batches and matrices too, which the packed f32 kernel serves faster."""
    ctx.set_tuning("gemv_tc", 1)
    yield
    ctx.set_tuning("gemv_tc", 0)


@pytest.mark.parametrize("m,k,batch", [(1, 256, 2), (127, 512, 8), (128, 256, 3), (129, 1280, 4), (1000, 2560, 5), (300, 18944, 8), (19100, 768, 7), (40, 5376, 6)])
def test_batched_q8_0(ctx, oracle, on_tc, m, k, batch):
    import runit_mac_b200 as R
    O = oracle
    rng = np.random.default_rng(m + k + batch)
    w = O.rand_weights(0, rng, m, k)
    x = (rng.normal(0, 1, (batch, k)) * 10.0 ** rng.uniform(-2, 2, (batch, 1))).astype(np.float32)
    x[0, 3] = 4000.0
    x[1, :256] = 0
    res = rng.normal(0, 1, (batch, m)).astype(np.float32)
    ref = O.gemv(0, w, x, m, k, O.TIER_F64)
    wb, xb, yb = ctx.buffer_from(w), ctx.buffer_from(x), ctx.new_buffer(batch * m * 4)
    outs = []
    for r in (None, res, None):
        R.gemv_batched_f32(ctx, 0, wb, xb, yb, None if r is None else ctx.buffer_from(r), m, k, batch)
        ctx.flush()
        outs.append(yb.download(np.float32, batch * m))
    for n in range(batch):
        at = slice(n * m, (n + 1) * m)
        assert_close(O, ref.reshape(-1)[at], outs[0][at], rel_tol=2e-5, what="row %d" % n)
        assert_close(O, ref.reshape(-1)[at] + res[n], outs[1][at], rel_tol=2e-5, what="row %d with residual" % n)
    assert np.array_equal(outs[0], outs[2])
    ctx.set_tuning("gemv_math", 1)                  # the packed f32 kernel
    try:
        R.gemv_batched_f32(ctx, 0, wb, xb, yb, None, m, k, batch)
        ctx.flush()
    finally:
        ctx.set_tuning("gemv_math", 0)
    for n in range(batch):
        assert_close(O, yb.download(np.float32, batch * m)[n * m:(n + 1) * m], outs[0][n * m:(n + 1) * m], rel_tol=2e-5, what="against packed f32")


@pytest.mark.parametrize("k", [256, 1536, 3584])
def test_batched_q8_0_bits_do_not_depend_on_the_launch(ctx, oracle, on_tc, k):
    """A matrix alone, in one launch with two others, and as the first rows of a larger one: the same bits."""
    import runit_mac_b200 as R
    O = oracle
    rows, batch = (700, 128, 2000), 6
    rng = np.random.default_rng(k)
    ws = [O.rand_weights(0, rng, m, k) for m in rows]
    xb = ctx.buffer_from(rng.normal(0, 1, (batch, k)).astype(np.float32))
    wb = [ctx.buffer_from(w) for w in ws]
    outs = [ctx.new_buffer(batch * m * 4) for m in rows]
    R.gemv_batched_multi_f32(ctx, 0, wb, xb, outs, rows, k, batch)
    both = ctx.buffer_from(np.concatenate([ws[0].reshape(rows[0], -1)[:640], ws[2].reshape(rows[2], -1)]))
    large, single = ctx.new_buffer(batch * 2640 * 4), ctx.new_buffer(batch * 2000 * 4)
    R.gemv_batched_f32(ctx, 0, both, xb, large, None, 2640, k, batch)
    ctx.flush()
    for b1, m, o in zip(wb, rows, outs):
        R.gemv_batched_f32(ctx, 0, b1, xb, single, None, m, k, batch)
        ctx.flush()
        assert np.array_equal(single.download(np.float32, batch * m), o.download(np.float32, batch * m))
    large = large.download(np.float32, batch * 2640).reshape(batch, 2640)
    assert np.array_equal(large[:, :640], outs[0].download(np.float32, batch * 700).reshape(batch, 700)[:, :640])
    assert np.array_equal(large[:, 640:], outs[2].download(np.float32, batch * 2000).reshape(batch, 2000))


def test_batched_q8_0_value_that_is_not_finite_stays_with_its_row(ctx, oracle, on_tc):
    import runit_mac_b200 as R
    O = oracle
    m, k, batch = 200, 1024, 5
    rng = np.random.default_rng(5)
    w = O.rand_weights(0, rng, m, k)
    x = rng.normal(0, 1, (batch, k)).astype(np.float32)
    x[1, 700], x[3, 0] = np.inf, np.nan
    yb = ctx.new_buffer(batch * m * 4)
    R.gemv_batched_f32(ctx, 0, ctx.buffer_from(w), ctx.buffer_from(x), yb, None, m, k, batch)
    ctx.flush()
    got = yb.download(np.float32, batch * m).reshape(batch, m)
    assert not np.isfinite(got[[1, 3]]).any()
    for n in (0, 2, 4):
        assert_close(O, O.gemv(0, w, x[n], m, k, O.TIER_F64), got[n], rel_tol=2e-5, what="row %d" % n)


@pytest.mark.parametrize("counts", [(0, 1, 7, 8, 9, 16, 17, 30),            # groups of 8 columns
                                    (0, 1, 15, 16, 17, 48, 49, 97)])        # groups of 48 in tiles of 16
@pytest.mark.parametrize("h,ff", [(256, 256), (1280, 768)])
def test_moe_slots_per_expert(ctx, oracle, counts, h, ff):
    """Slots of an expert around the tiles' and the groups' sizes; the router picks by one large activation."""
    import runit_mac_b200 as R
    O = oracle
    E = len(counts)
    expert = np.repeat(np.arange(E), counts)
    T = len(expert)
    rng = np.random.default_rng(T + h)
    rng.shuffle(expert)
    weights = [O.rand_q4k(rng, E * r, c) for r, c in ((ff, h), (ff, h), (h, ff))]
    router = np.zeros((E, h), np.float32)
    router[np.arange(E), np.arange(E)] = 8.0
    x = rng.normal(0, 1, (T, h)).astype(np.float32)
    x[:, :E] = 0
    x[np.arange(T), expert] = 4.0
    res = rng.normal(0, 1, (T, h)).astype(np.float32)
    ref, ridx, _ = O.moe_layer_q4k(router, *weights, x, h=h, ff=ff, E=E, top_k=1, renorm=False, residual=res)
    got, idx = run(ctx, R, [ctx.buffer_from(a) for a in (router, *weights)], x, res, h, ff, E, 1)
    assert (idx[:, 0] == expert).all() and (ridx[:, 0] == expert).all()
    assert_close(O, ref, got, rel_tol=2e-5, what="slots per expert")


@pytest.mark.parametrize("m,k", [(8192, 256), (8193, 512), (8199, 14336), (37889, 256), (18944, 512), (18945, 512), (18951, 768), (38008, 768), (40001, 3584), (38023, 1280), (37960, 1792), (38000, 2560), (40016, 3584), (37904, 8192)])
def test_q6k(ctx, oracle, m, k):
    """Rows of odd and even counts of 210-byte superblocks (a row's first byte modulo 16 takes every even value, or a few), a last tile of 8 to 120
    rows, 1 to 7 rows behind the last group of eight, a matrix that ends in the middle of a word; with and without a residual, in place."""
    import torch
    import runit_mac_b200 as R
    O = oracle
    nb = k // 256
    g = torch.Generator(device="cuda").manual_seed(m)
    w = torch.randint(0, 256, (m * nb, 210), generator=g, device="cuda", dtype=torch.uint8)
    w[:, 208:210] = (torch.rand(m * nb, generator=g, device="cuda") + 0.5).half().view(torch.uint8).reshape(-1, 2)
    x = torch.randn(k, generator=g, device="cuda")
    x[5] = 500.0
    res = torch.randn(m, generator=g, device="cuda") * 100
    y = torch.zeros(2, m, device="cuda")
    old = torch.zeros(m, device="cuda")
    z = res.clone()
    torch.cuda.synchronize()
    R.gemv_q6k_f32in_f32out(ctx, w, x, y[0], m, k)
    R.gemv_q6k_f32in_f32out(ctx, w, x, y[1], m, k)
    R.gemv_q6k_add_f32_f32in(ctx, w, x, z, z, m, k)
    ctx.set_tuning("kquant_variant", 2)             # the tile kernel, with f32 products
    try:
        R.gemv_q6k_f32in_f32out(ctx, w, x, old, m, k)
    finally:
        ctx.set_tuning("kquant_variant", 0)
    ctx.flush()
    assert torch.equal(y[0], y[1])
    assert_close(O, old.cpu().numpy(), y[0].cpu().numpy(), rel_tol=2e-5, what="against packed f32")
    rows = torch.cat([torch.arange(200), torch.arange(m - 200, m), torch.randint(0, m, (100,))])
    ref = O.gemv(5, w.reshape(m, -1)[rows.cuda()].cpu().numpy(), x.cpu().numpy(), len(rows), k, O.TIER_F64)
    assert_close(O, ref, y[0][rows.cuda()].cpu().numpy(), rel_tol=2e-5, what="q6k")
    assert_close(O, ref + res[rows.cuda()].double().cpu().numpy(), z[rows.cuda()].cpu().numpy(), rel_tol=2e-5, what="q6k with residual")


@pytest.mark.parametrize("fmt", [0, 5])
def test_infinities_and_nan(ctx, oracle, on_tc, fmt):
    """An infinite activation gives infinities of the weights' signs (NaN where the weight is 0), a NaN gives NaN, in its own row of activations."""
    import torch
    import runit_mac_b200 as R
    O = oracle
    m, k, batch = (19200, 768, 1) if fmt == 5 else (300, 768, 3)
    g = torch.Generator(device="cuda").manual_seed(fmt)
    if fmt == 5:
        w = torch.randint(0, 256, (m * k // 256, 210), generator=g, device="cuda", dtype=torch.uint8)
        w[:, 208:210] = (torch.rand(len(w), generator=g, device="cuda") + 0.5).half().view(torch.uint8).reshape(-1, 2)
    else:
        w = torch.randint(0, 256, (m * k // 32, 34), generator=g, device="cuda", dtype=torch.uint8)
        w[:, :2] = (torch.rand(len(w), generator=g, device="cuda") + 0.5).half().view(torch.uint8).reshape(-1, 2)
    for at, value in (([300], float("inf")), ([300], float("-inf")), ([10], float("nan")), ([0, 700], float("inf"))):
        x = torch.randn(batch, k, generator=g, device="cuda")
        x[batch - 1, at] = value
        y = torch.zeros(batch, m, device="cuda")
        torch.cuda.synchronize()
        if fmt == 5:
            R.gemv_q6k_f32in_f32out(ctx, w, x, y, m, k)
        else:
            R.gemv_batched_f32(ctx, 0, w, x, y, None, m, k, batch)
        ctx.flush()
        assert torch.isfinite(y[:batch - 1]).all()
        got = y[batch - 1].cpu().numpy()
        assert not np.isfinite(got).any()
        with np.errstate(invalid="ignore"):
            ref = O.gemv(fmt, w.reshape(m, -1)[:300].cpu().numpy(), x[batch - 1].cpu().numpy(), 300, k, O.TIER_F64).reshape(-1)
        assert np.array_equal(got[:300], ref.astype(np.float32), equal_nan=True)


def rms_error(got, ref):
    return ((got.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("k", [256, 1792, 3584])
@pytest.mark.parametrize("fmt", [0, 5])
def test_error_is_that_of_f32_products_at_most(ctx, oracle, on_tc, fmt, k, heavy):
    """Against 64 bits, over rows enough that the root mean square stands to a few per cent, with activations as they come and with a few channels that
    dominate, as hidden states of large models have.  (A tenth of room: it lies 10 to 40 % below.)"""
    import torch
    import runit_mac_b200 as R
    m, batch, block = 8192, 1 if fmt else 4, 210 if fmt else 34
    g = torch.Generator(device="cuda").manual_seed(k)
    w = torch.randint(0, 256, (m * k // (256 if fmt else 32), block), generator=g, device="cuda", dtype=torch.uint8)
    at = 208 if fmt else 0
    w[:, at:at + 2] = (torch.rand(len(w), generator=g, device="cuda") + 0.5).half().view(torch.uint8).reshape(-1, 2)
    x = torch.randn(batch, k, generator=g, device="cuda")
    if heavy:
        x *= torch.exp(torch.randn(batch, k, generator=g, device="cuda"))
        x[:, ::200] *= 100
    values = torch.from_numpy(oracle.dequant_rows(fmt, w.cpu().numpy(), m, k)).cuda().double()      # f16 times small integers: exact in f32
    ref = x.double() @ values.T
    errors = []
    for f32 in (False, True):
        ctx.set_tuning("gemv_math", int(f32))
        ctx.set_tuning("kquant_variant", 2 * f32)
        ctx.set_tuning("kquant_prepare", 2 * f32)
        y = torch.zeros(batch, m, device="cuda")
        torch.cuda.synchronize()
        try:
            if fmt:
                R.gemv_q6k_f32in_f32out(ctx, w, x, y, m, k)
            else:
                R.gemv_batched_f32(ctx, 0, w, x, y, None, m, k, batch)
            ctx.flush()
        finally:
            for key in ("gemv_math", "kquant_variant", "kquant_prepare"):
                ctx.set_tuning(key, 0)
        errors.append(rms_error(y, ref))
    assert errors[0] <= 1.1 * errors[1], errors


@pytest.mark.parametrize("T,most", [(32, 9.0e-7), (96, 1.9e-6)])
def test_error_of_the_sorted_moe_layer(ctx, oracle, T, most):
    """Groups of 8 and of 48 slots against 64 bits: below what the products measured with mma.sync (most), because the sums that the tensor cores cut off
    are kept short or small."""
    import torch
    import runit_mac_b200 as R
    E, k, h, ff = 8, 2, 1024, 512
    rng = np.random.default_rng(T)
    router, x = rng.normal(0, 0.02, (E, h)).astype(np.float32), rng.normal(0, 1, (T, h)).astype(np.float32)
    weights = [oracle.rand_q4k(rng, E * r, c) for r, c in ((ff, h), (ff, h), (h, ff))]
    out, idx, w = ctx.new_buffer(T * h * 4), ctx.new_buffer(T * k * 4), ctx.new_buffer(T * k * 4)
    nbytes = R.moe_scratch_bytes(ctx, T, h, ff, E, k)
    scratch = ctx.new_buffer(nbytes)
    bufs = [ctx.buffer_from(a) for a in (router, *weights, x)]
    ctx.set_tuning("moe_slots", 1)
    try:
        R.moe_layer_q4k(ctx, *bufs, None, out, idx, w, scratch, nbytes, T, h, ff, E, k, 0)
        ctx.flush()
    finally:
        ctx.set_tuning("moe_slots", 0)
    gate, up, down = (torch.from_numpy(oracle.dequant_rows(2, a, E * r, c)).cuda().double().reshape(E, r, c) for a, (r, c) in zip(weights, ((ff, h), (ff, h), (h, ff))))
    idx, w = (torch.from_numpy(b.download(t, T * k).reshape(T, k)).cuda() for b, t in ((idx, np.int32), (w, np.float32)))
    xd, ref = torch.from_numpy(x).cuda().double(), torch.zeros(T, h, device="cuda", dtype=torch.float64)
    for e in range(E):
        t, i = torch.nonzero(idx == e, as_tuple=True)
        act = torch.nn.functional.silu(xd[t] @ gate[e].T) * (xd[t] @ up[e].T)
        ref.index_add_(0, t, w[t, i, None].double() * (act @ down[e].T))
    error = rms_error(torch.from_numpy(out.download(np.float32, T * h).reshape(T, h)).cuda(), ref)
    assert error <= most, error
