"""The tcgen05 matvecs, folded and canonical, read an ARPACK-order vector
themselves where no projector asks for the planar one.  Against the general way (a projector of
weight 0 takes it): the same operands, so the same numbers, over sectors
around the 64 rows and 8 or 32 columns of their tiles, odd sizes, classes of one and
of several states and bonds whose sectors lie in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bond(rng, dims, shuffled):
    q = np.repeat(np.arange(len(dims)), dims)
    if shuffled:
        rng.shuffle(q)
    return q.reshape(-1, 1).astype(np.int64)


@pytest.mark.parametrize("left,right,charges,shuffled", [
    ([63, 64, 65], [7, 8, 9], [0], False),
    ([1, 129, 2, 127], [1, 17, 5], [0, 1, 1], True),
    ([10, 33, 66], [31, 3, 8, 64], [0, 0, 1, 1, 1, 2], True),
])
def test_reads_arpack_vector(left, right, charges, shuffled):
    from chainamps_b200 import (Context, TwoVertexComponents, models, CMPS_SPLIT_TF32, CMPS_SPLIT_BF16,
                                CMPS_ORDER_FOLDED, CMPS_ORDER_CANONICAL, CMPS_FORM_CANONICAL_TC)
    rng = np.random.default_rng(len(left) + len(charges))
    d, D, rules = len(charges), 3, (0,)
    ch, bq = np.array(charges, np.int64).reshape(-1, 1), np.zeros((D, 1), np.int64)
    bl, br = _bond(rng, left, shuffled), _bond(rng, right, shuffled)
    W = rng.standard_normal((d, D, d, D)) + 1j * rng.standard_normal((d, D, d, D))
    W = W * (ch[:, 0][:, None] == ch[:, 0][None, :]).astype(float)[:, None, :, None]
    L = models.random_environment(rng, rules, bl, bq, list(range(D)), right=False)
    R = models.random_environment(rng, rules, br, bq, list(range(D)), right=True)
    ctx = Context(0)
    h = TwoVertexComponents(ctx, rules, L, models.mpo_tensor(ch, W, bq), R)
    x = rng.standard_normal(h.n) + 1j * rng.standard_normal(h.n)
    for order, precision in ((CMPS_ORDER_FOLDED, CMPS_SPLIT_TF32), (CMPS_ORDER_FOLDED, CMPS_SPLIT_BF16),
                             (CMPS_ORDER_CANONICAL, CMPS_SPLIT_BF16)):
        h.set_order(order)
        h.set_precision(precision)
        assert (h.split_form() == CMPS_FORM_CANONICAL_TC) == (order == CMPS_ORDER_CANONICAL)
        got = h.multiply(x)
        h.set_projectors([x], [0.0])
        want = h.multiply(x)
        h.set_projectors([], [])
        assert np.linalg.norm(want) > 0
        assert np.array_equal(got, want)
    del h
    ctx.close()
