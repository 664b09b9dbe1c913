"""The grouped FP64 GEMM at the edges of its tiles: sector dimensions one off
every slice and tile boundary (8, 16, 32, 64), K around the 16-value stage
and the 128-value fold, tasks of a single row or column -- through both
contraction orders, with complex and with real MPO entries (the real-A form).

The forward error of a stage is at most 2 (kFold + K / kFold + 6) u times the
product of the operands' absolute values (u = 2^-53; the factor 2 for the
three-multiplication imaginary part), under 300 u for K up to 2000; four
stages and the oracle's own sums stay under 1500 u of the matvec taken with
absolute values throughout."""
import numpy as np
import pytest

from oracle import blocks as ob

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LEFT = [1, 2, 7, 8, 9, 15, 17, 31, 33, 64, 65, 129]
RIGHT = [130, 5, 63, 32, 16, 8, 40, 1, 24, 3, 96, 10]


def _bond(dims):
    return np.repeat(np.arange(len(dims)), dims).reshape(-1, 1).astype(np.int64)


def _mats(t, chi, D):
    return ob.env_matrices(chi, D, t.colptr, t.rowind, t.values)


@pytest.mark.parametrize("d,real_w", [(1, False), (3, False), (3, True), (17, True)])
def test_matvec_at_tile_edges(d, real_w):
    from chainamps_b200 import (Context, TwoVertexComponents, models, CMPS_ORDER_FOLDED, CMPS_ORDER_CANONICAL)
    D, rules = 3, (0,)
    rng = np.random.default_rng(d)
    bl, br = (_bond(LEFT), _bond(RIGHT)) if d < 17 else (_bond(LEFT[:6]), _bond(RIGHT[3:9]))
    ch, bq = np.zeros((d, 1), np.int64), np.array([[0], [1], [-1]], np.int64)
    W = rng.standard_normal((d, D, d, D)) + (0 if real_w else 1j) * rng.standard_normal((d, D, d, D))
    # an entry conserves charge: q(b) = q(b') as the states carry none
    W = W * (bq[:, 0][None, :, None, None] == bq[:, 0][None, None, None, :]).astype(float)
    W = W.astype(np.complex128)
    L = models.random_environment(rng, rules, bl, bq, list(range(D)), right=False)
    R = models.random_environment(rng, rules, br, bq, list(range(D)), right=True)
    lm, rm = _mats(L, bl.shape[0], D), _mats(R, br.shape[0], D)
    ref = ob.BlockHeff(rules, ch, bl, br, bq, W, lm, rm)
    mag = ob.BlockHeff(rules, ch, bl, br, bq, np.abs(W).astype(np.complex128),
                       *[[None if m is None else np.abs(m).astype(np.complex128) for m in e] for e in (lm, rm)])
    x = rng.standard_normal(ref.n) + 1j * rng.standard_normal(ref.n)
    want, bound = ref.matvec(x), 1500 * U * np.abs(mag.matvec(np.abs(x).astype(np.complex128)))
    ctx = Context(0)
    h = TwoVertexComponents(ctx, rules, L, models.mpo_tensor(ch, W, bq), R)
    for order in (CMPS_ORDER_FOLDED, CMPS_ORDER_CANONICAL):
        h.set_order(order)
        err = np.abs(h.multiply(x) - want)
        assert np.all(err <= bound), (order, np.max(err / np.maximum(bound, 1e-300)))
    del h
    ctx.close()


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_folded_order_skips_zero_parts_of_t(seed):
    """Sparse MPOs in the folded order: slots that no LeftPart block produces,
    slots that no RightPart block reads, states that a slot connects on one
    side only, neighbouring states alike and unlike -- the rows and columns
    of T that the plans leave out.  FP64 as above; the split forms within
    2e-4 of the largest entry, as the other split tests at these sizes."""
    from chainamps_b200 import (Context, TwoVertexComponents, models, CMPS_FP64, CMPS_SPLIT_TF32, CMPS_SPLIT_BF16,
                                CMPS_ORDER_FOLDED)
    d, D, rules = 5, 6, (0,)
    rng = np.random.default_rng(seed)
    bl, br = _bond([9, 33, 1, 17]), _bond([40, 8, 3, 21])
    ch, bq = np.zeros((d, 1), np.int64), np.zeros((D, 1), np.int64)
    W = rng.standard_normal((d, D, d, D)) + 1j * rng.standard_normal((d, D, d, D))
    W = W * (rng.random((d, D, d, D)) < 0.06)
    W[:, :, :, 2] = 0     # produced by nothing
    W[:, 3] = 0           # read by nothing
    W[0, 0, 0, 0] = 1.0   # never empty
    L = models.random_environment(rng, rules, bl, bq, list(range(D)), right=False)
    R = models.random_environment(rng, rules, br, bq, list(range(D)), right=True)
    lm, rm = _mats(L, bl.shape[0], D), _mats(R, br.shape[0], D)
    ref = ob.BlockHeff(rules, ch, bl, br, bq, W, lm, rm)
    mag = ob.BlockHeff(rules, ch, bl, br, bq, np.abs(W).astype(np.complex128),
                       *[[None if m is None else np.abs(m).astype(np.complex128) for m in e] for e in (lm, rm)])
    x = rng.standard_normal(ref.n) + 1j * rng.standard_normal(ref.n)
    want, bound = ref.matvec(x), 1500 * U * np.abs(mag.matvec(np.abs(x).astype(np.complex128)))
    ctx = Context(0)
    for prec in (CMPS_FP64, CMPS_SPLIT_TF32, CMPS_SPLIT_BF16):
        h = TwoVertexComponents(ctx, rules, L, models.mpo_tensor(ch, W, bq), R)
        h.set_order(CMPS_ORDER_FOLDED)
        h.set_precision(prec)
        err = np.abs(h.multiply(x) - want)
        assert np.all(err <= (bound if prec == CMPS_FP64 else 2e-4 * np.max(np.abs(want)))), (prec, np.max(err))
        del h
    ctx.close()


@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("ratio", [1e-4, 1e-8, 1e-12])
def test_small_component_keeps_its_accuracy(ratio, turned):
    """Nearly real operands (imaginary parts `ratio` of the real ones), and a
    vector turned by i: the small component of the result is as accurate as
    the large one.  Re and Im of a product are bounded each by its own terms,
    Re by |a||c| + |b||d| and Im by |a||d| + |b||c|, which is the product of
    |a| + j|b| and |c| + j|d| with j^2 = 1; a matvec of such numbers is two
    real ones, of the sums and of the differences of the two parts.  1500 u of
    it as above."""
    from chainamps_b200 import (Context, TwoVertexComponents, models, CMPS_ORDER_FOLDED, CMPS_ORDER_CANONICAL)
    d, D, rules = 3, 3, (0,)
    rng = np.random.default_rng(17)
    dims = ([9, 33, 64, 130], [65, 8, 3, 97])
    bl, br = _bond(dims[0]), _bond(dims[1])
    ch, bq = np.zeros((d, 1), np.int64), np.zeros((D, 1), np.int64)
    draw = lambda *s: rng.standard_normal(s) + 1j * ratio * rng.standard_normal(s)  # noqa: E731
    W = draw(d, D, d, D)
    L = models.random_environment(rng, rules, bl, bq, list(range(D)), right=False)
    R = models.random_environment(rng, rules, br, bq, list(range(D)), right=True)
    for t in (L, R):
        t.values = draw(t.values.size)
    lm, rm = _mats(L, bl.shape[0], D), _mats(R, br.shape[0], D)
    ref = ob.BlockHeff(rules, ch, bl, br, bq, W, lm, rm)
    x = draw(ref.n) * (1j if turned else 1.0)
    want = ref.matvec(x)

    def real_part(sign):
        f = lambda a: (np.abs(a.real) + sign * np.abs(a.imag)).astype(np.complex128)  # noqa: E731
        h = ob.BlockHeff(rules, ch, bl, br, bq, f(W), *[[None if m is None else f(m) for m in e] for e in (lm, rm)])
        return h.matvec(f(x)).real
    plus, minus = real_part(1.0), real_part(-1.0)
    bound_re, bound_im = 750 * U * (plus + minus), 750 * U * (plus - minus)
    ctx = Context(0)
    h = TwoVertexComponents(ctx, rules, L, models.mpo_tensor(ch, W, bq), R)
    for order in (CMPS_ORDER_FOLDED, CMPS_ORDER_CANONICAL):
        h.set_order(order)
        err = h.multiply(x) - want
        assert np.all(np.abs(err.real) <= bound_re), (order, np.max(np.abs(err.real) / bound_re))
        assert np.all(np.abs(err.imag) <= bound_im), (order, np.max(np.abs(err.imag) / bound_im))
    del h
    ctx.close()


def test_infinite_component():
    """One entry, x = inf + i, L = 2 + i, R = 1 - i: L x = inf + i inf and Re of
    its product with R is inf + inf."""
    from chainamps_b200 import Context, TwoVertexComponents, models
    one, z = np.zeros((1, 1), np.int64), np.ones((1, 1, 1, 1), np.complex128)
    rng, rules = np.random.default_rng(0), (0,)
    L = models.random_environment(rng, rules, one, one, [0], right=False)
    R = models.random_environment(rng, rules, one, one, [0], right=True)
    L.values, R.values = np.array([2 + 1j]), np.array([1 - 1j])
    ctx = Context(0)
    h = TwoVertexComponents(ctx, rules, L, models.mpo_tensor(one, z, one), R)
    got = h.multiply(np.array([complex(np.inf, 1.0)]))
    assert got[0].real == np.inf
    del h
    ctx.close()


PRECISIONS = ["CMPS_FP64", "CMPS_SPLIT_TF32", "CMPS_SPLIT_BF16"]


@pytest.mark.parametrize("precision", PRECISIONS)
def test_zero_operator(precision):
    """One MPO entry, into a slot that no entry leaves: H = 0, and no element of T
    is both produced and read."""
    import chainamps_b200 as ca
    from chainamps_b200 import models
    rng, rules = np.random.default_rng(4), (0,)
    bl, br, bq = _bond([5, 9]), _bond([8, 3]), np.zeros((2, 1), np.int64)
    W = np.zeros((1, 2, 1, 2), np.complex128)
    W[0, 0, 0, 1] = 1.0
    L = models.random_environment(rng, rules, bl, bq, [0, 1], right=False)
    R = models.random_environment(rng, rules, br, bq, [0, 1], right=True)
    ctx = ca.Context(0)
    h = ca.TwoVertexComponents(ctx, rules, L, models.mpo_tensor(np.zeros((1, 1), np.int64), W, bq), R)
    h.set_order(ca.CMPS_ORDER_FOLDED)
    h.set_precision(getattr(ca, precision))
    x = rng.standard_normal(h.n) + 1j * rng.standard_normal(h.n)
    assert np.array_equal(h.multiply(x), np.zeros(h.n))
    del h
    ctx.close()


@pytest.mark.parametrize("precision", PRECISIONS)
def test_owned_sector_that_nothing_reaches(precision):
    """States of charge 0 and 1, the MPO acts on charge 0 only.  In the sector of
    middle charge 0 the left vertex can carry charge 0 but the right one
    cannot: its rows of T are produced, none of its columns are read.  Owned
    alone, each sector is what it is in the whole matvec."""
    import torch
    import chainamps_b200 as ca
    from chainamps_b200 import models
    rng, rules = np.random.default_rng(5), (0,)
    ch, bq = np.array([[0], [1]], np.int64), np.zeros((1, 1), np.int64)
    W = np.zeros((2, 1, 2, 1), np.complex128)
    W[0, 0, 0, 0] = 1.0
    bl, br = _bond([4, 6]), _bond([7, 5]) + 1
    L = models.random_environment(rng, rules, bl, bq, [0], right=False)
    R = models.random_environment(rng, rules, br, bq, [0], right=True)
    ctx = ca.Context(0)
    h = ca.TwoVertexComponents(ctx, rules, L, models.mpo_tensor(ch, W, bq), R)
    h.set_order(ca.CMPS_ORDER_FOLDED)
    h.set_precision(getattr(ca, precision))
    x = torch.randn(h.n, dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    vin, vout = (torch.zeros(2 * h.n, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    h.theta_from_arpack_device(x.data_ptr(), vin.data_ptr(), 0)
    h.multiply_theta_device(vin.data_ptr(), vout.data_ptr(), 0)
    torch.cuda.synchronize()
    whole = vout.cpu().numpy().copy()
    base, _ = h.sector_table()
    seen = set()
    for m in range(len(base) - 1):
        own = np.zeros(len(base) - 1, np.uint8)
        own[m] = 1
        h.set_owned(own)
        vout.fill_(7.0)
        torch.cuda.synchronize()
        h.multiply_theta_device(vin.data_ptr(), vout.data_ptr(), 0)
        torch.cuda.synchronize()
        got, part = vout.cpu().numpy(), slice(base[m], base[m + 1])
        for plane in (0, h.n):
            assert np.array_equal(got[plane:][part], whole[plane:][part])
        seen.add(bool(np.any(whole[part])))
    assert seen == {True, False}
    del h
    ctx.close()
