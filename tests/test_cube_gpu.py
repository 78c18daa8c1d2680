"""The column-cube walks (four columns summed at once, rows in the classes of a
compiled shape) of FP64 x and split-dd: orders at the edges of the shape sizes
(no unused slot, up to three), sparse to dense shapes, shards, and the order
limits; against the CPU double-double oracle, the double-double kernel and a
product of smaller permanents, each within the walk's own error bound."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _real(n, d, seed, signed=False):
    """Density-d pattern with a hidden permutation, values (0, 1] or normal."""
    rng = np.random.default_rng([n, seed])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    return mask * (rng.standard_normal((n, n)) if signed else 1.0 - rng.random((n, n)))


def _check(engine, A, want, want_err, kernels):
    for variant in kernels:
        r = engine.exact_dense(A, variant=variant)
        assert r.kernel == variant
        # the bound is of the (hi, lo) pair; value rounds it once more
        tol = r.rel_error_estimate * abs(want) + want_err + U * abs(want)
        assert abs(r.value - want) <= tol, (variant, r.value, want, tol)
        parts = [engine.exact_dense_shard(A, s, 3, variant=variant) for s in range(3)]
        assert abs(sum(p.hi for p in parts) + sum(p.lo for p in parts) - r.value) <= 2 * tol + 4 * U * abs(want), variant


@pytest.mark.parametrize("n,d,signed", [(25, 0.12, False), (25, 0.5, True), (26, 0.95, False), (28, 0.35, False),
                                        (29, 0.7, False)])
def test_cube_vs_oracle_dd(engine, orc, pb, n, d, signed):
    A = _real(n, d, 1, signed)
    hi, lo = orc.perm_dd(A)
    r = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_SDD)
    # the oracle's own error: (4n + 32) u^2 sum|t|
    _check(engine, A, hi + lo, (4 * n + 32) * U * U * r.abs_term_sum,
           (pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_SDD))


@pytest.mark.parametrize("n,d", [(32, 0.5), (33, 0.25), (36, 0.2)])
def test_cube_vs_double_double_kernel(engine, pb, n, d):
    A = _real(n, d, 2)
    r = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_DD)
    _check(engine, A, r.hi + r.lo, (r.rel_error_estimate + U) * abs(r.value),
           (pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_SDD))


@pytest.mark.parametrize("n,k", [(40, 21), (37, 20)])
def test_cube_largest_orders_vs_product(engine, orc, pb, n, k):
    """Two diagonal blocks, rows and columns shuffled: the permanent is the
    product of the blocks'."""
    rng = np.random.default_rng(n)
    B, C = _real(k, 0.9, 3), _real(n - k, 0.9, 4)
    A = np.zeros((n, n))
    A[:k, :k], A[k:, k:] = B, C
    A = A[rng.permutation(n)][:, rng.permutation(n)]
    b, c = orc.perm_dd(B), orc.perm_dd(C)
    want = (b[0] + b[1]) * (c[0] + c[1])
    # each factor rounded once, and their product
    r = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE)
    assert abs(r.value - want) <= (r.rel_error_estimate + 4 * U) * want


def test_cube_transposed_and_permuted_inputs_agree(engine, pb):
    """The layout may walk the transpose: a matrix with sparse rows and its
    transpose (sparse columns) have one permanent."""
    rng = np.random.default_rng(11)
    n = 27
    A = _real(n, 0.85, 5)
    A[:4] *= rng.random((4, n)) < 0.3
    A[np.arange(4), np.arange(4)] = 1.0
    got = [engine.exact_dense(M, variant=pb.PERM_KERNEL_DENSE_SDD) for M in (A, A.T.copy(), A[::-1, ::-1].copy())]
    for g in got[1:]:
        assert abs(g.value - got[0].value) <= (g.rel_error_estimate + got[0].rel_error_estimate + 2 * U) * got[0].value


def _integers(n, d, top, seed, signed=False):
    rng = np.random.default_rng([n, seed, top])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    vals = rng.integers(1, top + 1, (n, n))
    return (mask * (vals * rng.choice([-1, 1], (n, n)) if signed else mask * vals)).astype(np.float64)


@pytest.mark.parametrize("n,d,top,signed", [(25, 0.12, 4, False), (25, 0.5, 1, False), (26, 0.4, 3, True),
                                            (27, 0.5, 4, False), (28, 0.7, 4, False), (29, 0.3, 1, False),
                                            # so few rows in the first chains that their products are exact
                                            (26, 0.05, 3, True),
                                            # row sums at the int32 runs' limit (four of about 215) and beyond it
                                            (25, 0.5, 33, False), (25, 0.5, 60, False)])
def test_cube_integer_walks_vs_exact(engine, orc, pb, n, d, top, signed):
    """int32 walks, FP64 and double-double products: against the exact
    multi-modular oracle within their bounds; shards add up."""
    A = _integers(n, d, top, 6, signed)
    want = float(orc.perm_exact_int(A)[0])
    _check(engine, A, want, U * abs(want), (pb.PERM_KERNEL_DENSE_INT, pb.PERM_KERNEL_DENSE_INT_DD))
    r = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_INT_DD)
    assert abs(r.value - want) <= 2 * U * abs(want) + r.rel_error_estimate * abs(want)


@pytest.mark.parametrize("n,k", [(36, 19), (33, 20)])
def test_cube_integer_walks_vs_product(engine, orc, pb, n, k):
    rng = np.random.default_rng(n)
    B, C = _integers(k, 0.8, 4, 7), _integers(n - k, 0.8, 4, 8)
    A = np.zeros((n, n))
    A[:k, :k], A[k:, k:] = B, C
    A = A[rng.permutation(n)][:, rng.permutation(n)]
    want = float(orc.perm_exact_int(B)[0] * orc.perm_exact_int(C)[0])
    for variant in (pb.PERM_KERNEL_DENSE_INT, pb.PERM_KERNEL_DENSE_INT_DD):
        r = engine.exact_dense(A, variant=variant)
        assert abs(r.value - want) <= (r.rel_error_estimate + 2 * U) * want, variant


def test_cube_walks_in_a_batch(engine, orc, pb):
    """From order 25 a batch's matrices walk in column cubes, by launches of
    their own beside the persistent kernel: values and error estimates in the
    caller's order, for real, binary and dense matrices mixed with small ones,
    the same on every run."""
    rng = np.random.default_rng(21)
    mats = []
    for n, d in ((12, 0.5), (25, 0.3), (26, 0.95), (9, 0.6), (27, 0.5), (25, 0.8), (28, 0.4), (24, 0.5)):
        mats += [_real(n, d, 31), _integers(n, d, 1, 32), _integers(n, d, 4, 33)]
    mats = [mats[i] for i in rng.permutation(len(mats))]
    b = engine.batch(mats)
    try:
        plain, _ = b.run()
        again, _ = b.run()
        values, estimates, _, _ = b.run_ex()
    finally:
        b.free()
    assert np.array_equal(plain, again)
    for M, p, v, e in zip(mats, plain, values, estimates):
        r = engine.exact_dense(M)
        assert abs(v - r.value) <= (e + r.rel_error_estimate + 2 * U) * abs(r.value), M.shape
        assert abs(p - r.value) <= 1e-10 * abs(r.value), M.shape


@pytest.mark.parametrize("n,d", [(19, 0.5), (20, 0.3), (20, 0.7), (21, 0.5), (24, 0.6), (22, 0.95)])
def test_whole_walks_with_own_term_sum(engine, orc, n, d):
    """Policy calls below order 25: value within the reported bound, and the
    sum of the absolute terms against direct evaluation."""
    A = _real(n, d, 17)
    r = engine.exact_dense(A)
    hi, lo = orc.perm_dd(A)[:2]
    assert abs(r.value - (hi + lo)) <= (r.rel_error_estimate + 2 * U) * abs(hi + lo)
    if n == 20:
        sign = 1.0 - 2.0 * ((np.arange(2 ** (n - 1))[:, None] >> np.arange(n - 1)) & 1)
        s1 = np.abs(np.prod(A[:, n - 1] + sign @ A[:, :n - 1].T, axis=1)).sum() * 2.0 ** (1 - n)
        # x carries n roundings, the product n more, either way
        assert abs(r.abs_term_sum - s1) <= 1e-9 * s1
