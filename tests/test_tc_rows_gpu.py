"""Packed rows times a few columns on tcgen05 (tc_rows.cuh): the MoE layer with its slots sorted by expert, at the edges of its tiles.

Bound: an activation keeps 22 bits (two f16 halves of x / 2^e, error <= 2^-22 of it or 2^-35 of the largest of its 256), products are exact, sums
are f32: 2^-24 of the running sum per addition along 32 products, 8 blocks and K / 256 units.  2e-5 of max(|ref|, rms) holds with room."""
import numpy as np
import pytest

from helpers import assert_close
from test_moe_slots_gpu import run

pytestmark = pytest.mark.gpu


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
