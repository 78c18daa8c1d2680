"""Rows and columns of different sizes in the column-cube walks.  A certified
walk may take the transpose, whose terms are larger without limit when the rows
differ in size; scaling rows or columns only multiplies the permanent."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _matrix(n, d, seed, values="real"):
    rng = np.random.default_rng([n, seed])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    v = 1.0 - rng.random((n, n)) if values == "real" else rng.integers(1, 4, (n, n)).astype(np.float64)
    return mask * v


SCALES = {"powers": lambda n: 10.0 ** -(np.arange(n) % 4), "every_other": lambda n: np.where(np.arange(n) % 2, 1e-3, 1.0)}


@pytest.mark.parametrize("n,seeds", [(25, 4), (29, 4), (32, 3), (36, 1)])
@pytest.mark.parametrize("scale", ["powers", "every_other"])
@pytest.mark.parametrize("axis", ["rows", "columns"])
def test_scaled_real_matrices(engine, pb, n, seeds, scale, axis):
    """Entries are rounded once by the scaling, so the permanent of a matrix
    without negative entries moves by n roundings at most."""
    s = SCALES[scale](n)
    for seed in range(seeds):
        A = _matrix(n, 0.5, seed)
        want = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_SDD)
        assert want.rel_error_estimate < 1e-15
        B = A * (s[:, None] if axis == "rows" else s[None, :])
        factor = float(np.prod(s, dtype=np.longdouble))
        for variant in (0, pb.PERM_KERNEL_DENSE_SDD):
            r = engine.exact_dense(B, variant=variant)
            assert r.rel_error_estimate < 1e-10, (seed, variant, r.kernel)
            tol = (n + 4) * U + r.rel_error_estimate + want.rel_error_estimate
            assert abs(r.value / factor / want.value - 1.0) <= tol, (seed, variant, r.kernel)


@pytest.mark.parametrize("n,axis", [(25, "rows"), (28, "rows"), (29, "rows"), (31, "rows"), (29, "columns"), (32, "columns")])
def test_scaled_integer_matrices(engine, pb, n, axis):
    """Powers of two, small enough for the int32 row products: exact."""
    s = np.where(np.arange(n) % 2, 8.0, 1.0)
    for seed in range(3):
        A = _matrix(n, 0.35, seed, "int")
        want = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_INT_DD)
        B = A * (s[:, None] if axis == "rows" else s[None, :])
        r = engine.exact_dense(B)
        assert r.kernel == pb.PERM_KERNEL_DENSE_INT_DD
        assert r.rel_error_estimate < 1e-10
        tol = 2 * U + r.rel_error_estimate + want.rel_error_estimate
        assert abs(r.value / np.prod(s) / want.value - 1.0) <= tol


@pytest.mark.parametrize("n", [25, 30])
def test_column_beyond_the_split_is_accepted(engine, pb, n):
    """Split-dd takes rows with absolute sums below 2^1020.  A column may add
    up to more: then the transpose is no choice, but the call is not refused
    (its terms overflow; the status is what is asked here)."""
    A = _matrix(n, 0.5, 1)
    A[:8, 0] = 2.0 ** 1018
    assert A.sum(axis=0).max() >= 2.0 ** 1020 > A.sum(axis=1).max()
    for variant in (pb.PERM_KERNEL_DENSE_SDD, 0):
        r = engine.exact_dense(A, variant=variant)
        assert r.kernel in (pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_DD, pb.PERM_KERNEL_DENSE_SDD)


@pytest.mark.parametrize("n", [21, 25, 29, 32])
def test_rows_of_extreme_sizes(engine, pb, n):
    """Rows times 2^200 and 2^-200 in turn: their products stay in range when
    rows are multiplied as they come, and would not when they are sorted into
    the classes of a cube.  Scaling is exact, so the permanent is too."""
    s = np.where(np.arange(n) % 2, 2.0 ** -200, 2.0 ** 200)
    factor = 2.0 ** (200 * (n % 2))
    for seed in range(3):
        A = _matrix(n, 0.5, seed)
        want = engine.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_SDD)
        for variant in (0, pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_SDD):
            r = engine.exact_dense(A * s[:, None], variant=variant)
            tol = 2 * U + r.rel_error_estimate + want.rel_error_estimate
            assert tol < 1e-8 and abs(r.value / factor / want.value - 1.0) <= tol, (seed, variant, r)


def test_rows_of_extreme_sizes_in_a_batch(engine):
    n = 26
    s = np.where(np.arange(n) % 2, 2.0 ** -200, 2.0 ** 200)
    mats = [_matrix(n, 0.5, seed) for seed in range(3)]
    b = engine.batch(mats + [A * s[:, None] for A in mats])
    try:
        for _ in range(2):
            values, estimates, _, _ = b.run_ex()
            for k in range(3):
                tol = 2 * U + estimates[k] + estimates[k + 3]
                assert tol < 1e-8 and abs(values[k + 3] / values[k] - 1.0) <= tol, k
    finally:
        b.free()
