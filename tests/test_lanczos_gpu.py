"""The Lanczos passes at the edges of their tiles and of their dispatch: odd
and even lengths (8- and 16-byte loads), lengths around one tile of 512, the
longer tiles of long vectors, more basis vectors than one launch of the
products takes (24), steps issued ahead (short vectors) and not, FP64 and
mixed precision.

H = A x 1 + 1 x B per sector with Hermitian A and B, so the lowest eigenvalue
is known.  The solver stops at a residual of tol max(1, |e|); the vector's
scaling and the recurrence's own rounding may add as much again, and the
eigenvalue is within the residual of one of H's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _hermitian(rng, n):
    m = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (m + m.conj().T) / np.sqrt(8 * n)


def _environment(mats, dims, slot, right):
    """Slot `slot` carries the sectors' matrices, the other one identities."""
    from chainamps_b200 import models
    chi = sum(dims)
    bond = np.repeat(np.arange(len(dims)), dims).reshape(-1, 1).astype(np.int64)
    bq, z = np.zeros((2, 1), np.int64), np.zeros((1, 1), np.int64)
    v = np.zeros((chi, 2, chi), np.complex128)
    v[:, 1 - slot] = np.eye(chi)
    at = 0
    for m in mats:
        v[at:at + len(m), slot, at:at + len(m)] = m
        at += len(m)
    S = models.MPXIndexSpec
    if right:
        return models.dense_to_tensor([S(False, False, bond), S(True, False, z), S(True, False, bq), S(False, False, z),
                                       S(True, False, bond), S(False, False, z)], 2, v.reshape(chi, 1, 2, 1, chi, 1))
    return models.dense_to_tensor([S(False, False, z), S(True, False, bond), S(True, False, z), S(False, False, bq),
                                   S(True, False, z), S(False, False, bond)], 3, v.reshape(1, chi, 1, 2, 1, chi))


@pytest.mark.parametrize("left,right,krylov,mixed", [
    ([13, 9], [11, 6], 24, False),          # n = 197, odd
    ([13, 9], [11, 6], 60, False),          # products in three launches
    ([16], [32], 25, False),                # one whole tile of 512; 24 + 1
    ([27], [19], 24, False),                # 513
    ([64, 31], [48, 40], 40, True),         # n = 4312, split BF16 steps
    ([601, 450], [701, 430], 40, False),    # n = 614801: long tiles, odd
    ([600, 450], [700, 430], 40, True),     # n = 613500: long tiles, even
    ([1100], [1000], 40, False),            # more than 2^20: not issued ahead
])
def test_lowest_eigenpair(left, right, krylov, mixed):
    from chainamps_b200 import Context, TwoVertexComponents, models, CMPS_FP64, CMPS_SPLIT_BF16
    rng = np.random.default_rng(sum(left) + krylov)
    A, B = [_hermitian(rng, n) for n in left], [_hermitian(rng, n) for n in right]
    want = min(np.linalg.eigvalsh(a)[0] + np.linalg.eigvalsh(b)[0] for a, b in zip(A, B))
    W = np.eye(2).reshape(1, 2, 1, 2).astype(np.complex128)
    Wt = models.mpo_tensor(np.zeros((1, 1), np.int64), W, np.zeros((2, 1), np.int64))
    ctx = Context(0)
    h = TwoVertexComponents(ctx, (0,), _environment(A, left, 0, False), Wt, _environment(B, right, 1, True))
    assert h.n == sum(a * b for a, b in zip(left, right))
    h.set_precision(CMPS_SPLIT_BF16 if mixed else CMPS_FP64)
    e, v, _ = h.HED(tol=TOL, max_restarts=200, krylov_dim=krylov)
    scale = max(1.0, abs(want))
    assert abs(e - want) <= 2 * TOL * scale
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-12
    h.set_precision(CMPS_FP64)
    assert np.linalg.norm(h.multiply(v) - e * v) <= 2 * TOL * scale
    st = h.eigs_stats()
    assert (st["split_matvecs"] > 0) == mixed
    del h
    ctx.close()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("left,right", [([1], [1]), ([1], [2]), ([1, 1], [1, 1])])
def test_smallest_spaces(left, right, mixed):
    """One and two entries: the Krylov space is the whole space, and with one
    entry the first step is the last one too."""
    from chainamps_b200 import Context, TwoVertexComponents, models, CMPS_FP64, CMPS_SPLIT_BF16
    rng = np.random.default_rng(7 * sum(left) + sum(right))
    A, B = [_hermitian(rng, n) for n in left], [_hermitian(rng, n) for n in right]
    want = min(np.linalg.eigvalsh(a)[0] + np.linalg.eigvalsh(b)[0] for a, b in zip(A, B))
    W = np.eye(2).reshape(1, 2, 1, 2).astype(np.complex128)
    Wt = models.mpo_tensor(np.zeros((1, 1), np.int64), W, np.zeros((2, 1), np.int64))
    ctx = Context(0)
    h = TwoVertexComponents(ctx, (0,), _environment(A, left, 0, False), Wt, _environment(B, right, 1, True))
    h.set_precision(CMPS_SPLIT_BF16 if mixed else CMPS_FP64)
    e, v, _ = h.HED(tol=TOL, max_restarts=200)
    scale = max(1.0, abs(want))
    assert abs(e - want) <= 2 * TOL * scale
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-12
    h.set_precision(CMPS_FP64)
    assert np.linalg.norm(h.multiply(v) - e * v) <= 2 * TOL * scale
    del h
    ctx.close()


@pytest.mark.parametrize("size,precision,canonical", [
    (1e120, "CMPS_FP64", False), (1e25, "CMPS_SPLIT_BF16", False), (1e25, "CMPS_SPLIT_TF32", False),
    (1e25, "CMPS_SPLIT_BF16", True), (1e25, "CMPS_SPLIT_TF32", True)])
@pytest.mark.parametrize("projected", [False, True])
def test_large_operators(size, precision, canonical, projected):
    """H of a size whose square still fits its format (64 bits, or the 32 of the
    split forms' operands), with and without a projector that lifts the
    ground state above the first excited one; tolerances as above."""
    import chainamps_b200 as ca
    from chainamps_b200 import models
    rng = np.random.default_rng(5)
    left, right = [13, 9], [11, 6]
    A, B = [[size * _hermitian(rng, n) for n in dims] for dims in (left, right)]
    levels = np.sort(np.concatenate([np.add.outer(np.linalg.eigvalsh(a), np.linalg.eigvalsh(b)).ravel()
                                     for a, b in zip(A, B)]))
    W = np.eye(2).reshape(1, 2, 1, 2).astype(np.complex128)
    Wt = models.mpo_tensor(np.zeros((1, 1), np.int64), W, np.zeros((2, 1), np.int64))
    ctx = ca.Context(0)
    h = ca.TwoVertexComponents(ctx, (0,), _environment(A, left, 0, False), Wt, _environment(B, right, 1, True))
    if canonical:
        h.set_order(ca.CMPS_ORDER_CANONICAL)
    if projected:
        _, ground, _ = h.HED(tol=TOL, max_restarts=200)
        h.set_projectors([ground.conj()], [2.0 * (levels[1] - levels[0])])
    want = levels[1 if projected else 0]
    h.set_precision(getattr(ca, precision))
    e, v, _ = h.HED(tol=TOL, max_restarts=200, krylov_dim=40)
    assert abs(e - want) <= 4 * TOL * abs(want)
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-12
    h.set_precision(ca.CMPS_FP64)
    assert np.linalg.norm(h.multiply(v) - e * v) <= 2 * TOL * abs(want)
    del h
    ctx.close()


def test_stats_count_dropped_steps():
    """A short vector's cycle that ends before its last step has issued one step
    more, whose matvec is part of the solve's time and of its counts."""
    from chainamps_b200 import Context, TwoVertexComponents, models
    rng = np.random.default_rng(3)
    left, right, krylov = [13, 9], [11, 6], 60
    A, B = [_hermitian(rng, n) for n in left], [_hermitian(rng, n) for n in right]
    W = np.eye(2).reshape(1, 2, 1, 2).astype(np.complex128)
    Wt = models.mpo_tensor(np.zeros((1, 1), np.int64), W, np.zeros((2, 1), np.int64))
    ctx = Context(0)
    h = TwoVertexComponents(ctx, (0,), _environment(A, left, 0, False), Wt, _environment(B, right, 1, True))
    _, _, applications = h.HED(tol=TOL, max_restarts=200, krylov_dim=krylov)
    st = h.eigs_stats()
    assert st["cycles"] == 1 and applications < krylov
    assert st["fp64_matvecs"] == applications + 1
    assert st["ms_fp64"] <= st["ms_total"]
    del h
    ctx.close()
