"""perm_cube_layout (host only): which calls walk column cubes; and, on the
GPU, that calls it answers -1 for walk the row layout the other queries name."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

U = 2.0 ** -53


def _matrix(n, d, seed, kind):
    rng = np.random.default_rng([n, seed, int(d * 100)])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    return mask * {"real": lambda: 1.0 - rng.random((n, n)), "bin": lambda: 1.0,
                   "int": lambda: rng.integers(1, 5, (n, n)) * 1.0}[kind]()


def _variants(pb, kind):
    return ((pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_SDD) if kind == "real" else
            (pb.PERM_KERNEL_DENSE_INT, pb.PERM_KERNEL_DENSE_INT_DD))


def test_orders_and_densities(pb):
    for kind in ("real", "bin", "int"):
        for variant in _variants(pb, kind):
            for n in (25, 28, 29, 32, 36, 37, 40):
                shape, ops = pb.cube_layout(_matrix(n, 0.4, 1, kind), variant)
                assert shape >= 0 and 100.0 < ops < 16 * 2 * n, (kind, variant, n)
                if variant != pb.PERM_KERNEL_DENSE_SDD:
                    assert pb.cube_layout(np.ones((n, n)), variant) == (-1, 0.0)
            # whole cubes begin at order 25 and end at 40
            for n in (1, 7, 20, 24, 41):
                assert pb.cube_layout(_matrix(n, 0.4, 1, kind), variant) == (-1, 0.0)
    A = _matrix(30, 0.4, 1, "real")
    for variant in (0, pb.PERM_KERNEL_DENSE_DD, pb.PERM_KERNEL_DENSE_SPLIT, pb.PERM_KERNEL_DENSE_TC, 99,
                    pb.PERM_KERNEL_DENSE_INT):  # not an integer matrix
        assert pb.cube_layout(A, variant) == (-1, 0.0)
    assert pb.load_library().perm_cube_layout(None, 30, pb.PERM_KERNEL_DENSE, None) == -1
    assert pb.load_library().perm_cube_layout(A.ctypes.data_as(ctypes.c_void_p), 65, pb.PERM_KERNEL_DENSE, None) == -1


def test_rows_of_different_sizes_and_infinities(pb):
    A = _matrix(30, 0.4, 2, "real")
    plain = pb.cube_layout(A, pb.PERM_KERNEL_DENSE)
    s = np.where(np.arange(30) % 2, 2.0 ** -300, 2.0 ** 300)
    assert pb.cube_layout(A * s[:, None], pb.PERM_KERNEL_DENSE) == plain
    B = A.copy()
    B[3, np.nonzero(B[3])[0][0]] = np.inf
    assert pb.cube_layout(B, pb.PERM_KERNEL_DENSE)[0] == -1
    # an entry that scaling would lose
    C = A * s[:, None]
    k = np.nonzero(C[0])[0]
    C[0, k[0]], C[0, k[1]] = 2.0 ** 900, 2.0 ** -900
    assert pb.cube_layout(C, pb.PERM_KERNEL_DENSE)[0] == -1


@pytest.mark.gpu
def test_calls_in_rows(engine, pb):
    """Matrices the cubes leave to row layouts of one, two and three levels."""
    found = set()
    for kind, densities in (("real", (0.8, 0.95)), ("bin", (0.6, 0.7, 0.8, 0.9)), ("int", (0.6, 0.7, 0.8, 0.9))):
        for n in (25, 27, 28, 30, 32):
            for d in densities:
                for seed in range(3):
                    A = _matrix(n, d, seed, kind)
                    for variant in _variants(pb, kind):
                        if pb.cube_layout(A, variant)[0] >= 0:
                            continue
                        if kind == "real":
                            r1, r2 = (pb.fp64_levels if variant == pb.PERM_KERNEL_DENSE else pb.sdd_levels)(A)
                            level = 3 if r1 else 2 if r2 else 1
                        else:
                            level = ((lambda g, ngo, ng1, ng2: 3 if ng1 else 2 if ngo else 1)(*pb.int_layout(A))
                                     if variant == pb.PERM_KERNEL_DENSE_INT else
                                     (lambda g, p, ngo, ng1, ng2: 3 if ng1 else 2 if ngo else 1)(*pb.intc_layout(A)))
                        if (kind, variant, level, n) in found:
                            continue
                        found.add((kind, variant, level, n))
                        r, rows = engine.exact_dense(A, variant=variant), engine.exact_dense_rows(A, variant=variant)
                        assert (r.hi, r.lo) == (rows.hi, rows.lo), (kind, variant, level, n)
                        want = engine.exact_dense(A, variant=_variants(pb, kind)[1])
                        tol = (r.rel_error_estimate + want.rel_error_estimate + 2 * U) * abs(want.value)
                        assert abs(r.value - want.value) <= tol
    levels = {f[:3] for f in found}
    for f in (("bin", pb.PERM_KERNEL_DENSE_INT, 3), ("bin", pb.PERM_KERNEL_DENSE_INT_DD, 2),
              ("bin", pb.PERM_KERNEL_DENSE_INT_DD, 3), ("int", pb.PERM_KERNEL_DENSE_INT_DD, 2),
              ("int", pb.PERM_KERNEL_DENSE_INT_DD, 3), ("real", pb.PERM_KERNEL_DENSE, 1),
              ("real", pb.PERM_KERNEL_DENSE_SDD, 1)):
        assert f in levels, (f, levels)
