"""Expert products with the slots sorted by expert (moe_slots.cu), through runit_moe_layer_q4k, against the oracle.

Bound: an activation keeps 22 bits (two f16 halves of x / 2^e, error <= 2^-22 of it or 2^-35 of the largest of its 256), products and the unpacked weights are
exact, sums are f32 over 256 weights and then over units.  With the 2^-24 of every f32 addition along h / 256 units and the
rounding of silu, 2e-5 of max(|ref|, rms) holds with room.  The launches per slot have 16-bit activations: up to 2^-15 of the
block's largest value in each of three products, 32 blocks' worth of which lie above the spread where a block holds an outlier;
they are held to the bar of the other tests of this layer (1e-3)."""
import numpy as np
import pytest

from helpers import assert_close

pytestmark = pytest.mark.gpu


def run(ctx, R, weights, x, res, h, ff, E, k, slots=1, piece=0):
    T = x.shape[0]
    nbytes = R.moe_scratch_bytes(ctx, T, h, ff, E, k)
    out, idx, w = ctx.new_buffer(T * h * 4), ctx.new_buffer(T * k * 4), ctx.new_buffer(T * k * 4)
    scratch = ctx.new_buffer(nbytes)
    ctx.set_tuning("moe_slots", slots)              # 1: small layers, too; 2: launches per slot
    ctx.set_tuning("moe_piece", piece)
    try:
        R.moe_layer_q4k(ctx, *weights, ctx.buffer_from(x), ctx.buffer_from(res), out, idx, w, scratch, nbytes, T, h, ff, E, k, 0)
        ctx.flush()
    finally:
        ctx.set_tuning("moe_slots", 0)
        ctx.set_tuning("moe_piece", 0)
    return out.download(np.float32, T * h).reshape(T, h), idx.download(np.int32, T * k).reshape(T, k)


# tokens around the threshold, tiles of 8 slots and groups of 32 (k = E: every expert has all tokens)
@pytest.mark.parametrize("T,h,ff,E,k", [(4, 256, 256, 8, 2), (8, 512, 256, 2, 2), (9, 256, 512, 2, 2), (32, 512, 256, 3, 3), (33, 256, 256, 2, 2),
                                        (41, 768, 512, 1, 1), (70, 512, 256, 40, 3), (130, 256, 256, 256, 4)])
def test_layer_matches_oracle(ctx, oracle, T, h, ff, E, k):
    import runit_mac_b200 as R
    O = oracle
    rng = np.random.default_rng(T * 1000 + E)
    router = rng.normal(0, 0.05, (E, h)).astype(np.float32)
    gate, up, down = (np.stack([O.rand_q4k(rng, r, c) for _ in range(E)]) for r, c in ((ff, h), (ff, h), (h, ff)))
    x = (rng.normal(0, 1, (T, h)) * 10.0 ** rng.uniform(-1, 1, (T, 1))).astype(np.float32)
    x[0, ::5] = 0
    x[1, :256] = 0                                  # a unit without a largest value
    x[2, 3] = 4000.0                                # one outlier: the rest of its unit keeps its precision
    res = rng.normal(0, 1, (T, h)).astype(np.float32)
    ref, ridx, _ = O.moe_layer_q4k(router, gate, up, down, x, h=h, ff=ff, E=E, top_k=k, renorm=False, residual=res)
    weights = [ctx.buffer_from(a) for a in (router, gate, up, down)]
    got, idx = run(ctx, R, weights, x, res, h, ff, E, k)
    same = (np.sort(idx, 1) == np.sort(ridx, 1)).all(1)
    assert same.sum() >= T - 1                      # at most one near tie
    assert_close(O, ref[same], got[same], rel_tol=2e-5, what="slots by expert")
    again, _ = run(ctx, R, weights, x, res, h, ff, E, k)
    assert (again == got).all()                     # the order of the slots inside an expert does not show
    pieces, _ = run(ctx, R, weights, x, res, h, ff, E, k, piece=7)      # several passes over one staging area
    assert_close(O, ref[same], pieces[same], rel_tol=2e-5, what="in pieces")
    per_slot, _ = run(ctx, R, weights, x, res, h, ff, E, k, slots=2)
    assert_close(O, ref[same], per_slot[same], what="launches per slot")


@pytest.mark.parametrize("T", [2, 12, 65])
def test_by_slot_gives_a_token_the_same_bits_at_every_size(ctx, oracle, T):
    """What INTEGRATION.md promises for prefill against decode; the sizes are those at which runit_moe_layer_q4k sorts, too."""
    import runit_mac_b200 as R
    O = oracle
    h, ff, E, k = 2048, 1024, 16, 4
    rng = np.random.default_rng(T)
    weights = [ctx.buffer_from(a) for a in [rng.normal(0, 0.05, (E, h)).astype(np.float32)] + [O.rand_q4k(rng, E * r, c) for r, c in ((ff, h), (ff, h), (h, ff))]]
    x, res = rng.normal(0, 1, (T, h)).astype(np.float32), rng.normal(0, 1, (T, h)).astype(np.float32)

    def layer(op, lo, hi):
        n = hi - lo
        out, nbytes = ctx.new_buffer(n * h * 4), R.moe_scratch_bytes(ctx, n, h, ff, E, k)
        op(ctx, *weights, ctx.buffer_from(x[lo:hi]), ctx.buffer_from(res[lo:hi]), out, None, None, ctx.new_buffer(nbytes), nbytes, n, h, ff, E, k, 0)
        ctx.flush()
        return out.download(np.float32, n * h).reshape(n, h)

    alone = np.concatenate([layer(R.moe_layer_q4k, t, t + 1) for t in range(T)])       # the decoding step's size
    assert np.array_equal(layer(R.moe_layer_q4k_by_slot, 0, T), alone)
    assert_close(O, alone, layer(R.moe_layer_q4k, 0, T), rel_tol=3e-4, what="sorted")


def test_outlier_without_weight(ctx, oracle):
    """An activation 2^18 times as large as the others of its unit, in a block whose weights are 0: what is left are the small ones, whose
    halves are off by 2^-35 of the largest at most, 2^-17 of a small one, in the mean square over the 512 a quarter of 2^-17 / sqrt(3): 1e-6,
    and five times that at the largest of the outputs."""
    import runit_mac_b200 as R
    O = oracle
    T, h, ff, E, k = 16, 512, 256, 2, 2
    rng = np.random.default_rng(16)

    def matrix(rows, cols, hole):
        nb = cols // 256
        d, dmin = np.abs(rng.normal(0, 0.003, (rows, nb))) + 1e-3, np.abs(rng.normal(0, 0.003, (rows, nb)))
        sc, mn = (rng.integers(0, 64, (rows, nb, 8), dtype=np.uint8) for _ in range(2))
        if hole:
            sc[:, 0, 0], mn[:, 0, 0] = 0, 0         # the unit's first block
        return O.pack_q4k(d, dmin, sc, mn, rng.integers(0, 16, (rows, nb, 256), dtype=np.uint8))

    router = rng.normal(0, 0.05, (E, h)).astype(np.float32)
    router[:, :32] = 0
    gate, up, down = (np.stack([matrix(r, c, c == h) for _ in range(E)]) for r, c in ((ff, h), (ff, h), (h, ff)))
    x = rng.normal(0, 1, (T, h)).astype(np.float32)
    x[:, 7] = 2.0 ** 18
    ref, _, _ = O.moe_layer_q4k(router, gate, up, down, x, h=h, ff=ff, E=E, top_k=k, renorm=False)
    got, _ = run(ctx, R, [ctx.buffer_from(a) for a in (router, gate, up, down)], x, np.zeros((T, h), np.float32), h, ff, E, k)
    assert_close(O, ref, got, rel_tol=2e-5, what="outlier without weight")


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("T", [8, 40])
def test_activation_that_is_not_finite_stays_with_its_token(ctx, oracle, T, bad):
    """One and several tiles per expert: the other columns of the token's tiles keep their bits, the token's output is not finite."""
    import runit_mac_b200 as R
    O = oracle
    h, ff, E, k = 512, 256, 2, 2                    # k = E: every expert has every token, whatever the router makes of the bad one
    rng = np.random.default_rng(T)
    weights = [ctx.buffer_from(a) for a in [rng.normal(0, 0.05, (E, h)).astype(np.float32)] + [O.rand_q4k(rng, E * r, c) for r, c in ((ff, h), (ff, h), (h, ff))]]
    x, res = rng.normal(0, 1, (T, h)).astype(np.float32), rng.normal(0, 1, (T, h)).astype(np.float32)
    clean, _ = run(ctx, R, weights, x, res, h, ff, E, k)
    x[3, 300] = bad
    got, _ = run(ctx, R, weights, x, res, h, ff, E, k)
    others = np.arange(T) != 3
    assert np.array_equal(got[others], clean[others]) and np.isfinite(clean).all()
    assert not np.isfinite(got[3]).any()


def test_built_in_scratch_gives_the_same_bits(ctx, oracle):
    """A size at which the slots are sorted and the intermediates fill a good part of the built-in region."""
    import runit_mac_b200 as R
    O = oracle
    T, h, ff, E, k = 48, 1024, 512, 16, 8
    rng = np.random.default_rng(48)
    weights = [ctx.buffer_from(a) for a in [rng.normal(0, 0.05, (E, h)).astype(np.float32)] + [O.rand_q4k(rng, E * r, c) for r, c in ((ff, h), (ff, h), (h, ff))]]
    x = ctx.buffer_from(rng.normal(0, 1, (T, h)).astype(np.float32))
    nbytes = R.moe_scratch_bytes(ctx, T, h, ff, E, k)
    assert nbytes <= ctx.lib.runit_moe_static_scratch_capacity()
    outs = [ctx.new_buffer(T * h * 4) for _ in range(2)]
    count = [ctx.launches]
    R.moe_layer_q4k(ctx, *weights, x, None, outs[0], None, None, ctx.new_buffer(nbytes), nbytes, T, h, ff, E, k, 0)
    count.append(ctx.launches)
    R.moe_layer_q4k_static(ctx, *weights, x, None, outs[1], None, None, T, h, ff, E, k, 0)
    count.append(ctx.launches)
    assert count[2] - count[1] == count[1] - count[0]
    ctx.flush()
    a, b = (o.download(np.float32, T * h) for o in outs)
    assert np.isfinite(a).all() and np.array_equal(a, b)
