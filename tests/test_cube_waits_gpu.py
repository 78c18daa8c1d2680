"""Failure detection in the column-cube launches, without a GPU fault: an
injected barrier that never completes makes the operand staging give up after
its limit; the call returns PERM_ETIMEOUT, and the context, its partial sums and
its ticket are as good as before."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _matrix(n, seed):
    rng = np.random.default_rng([n, seed])
    mask = (rng.random((n, n)) < 0.4) | (np.eye(n)[rng.permutation(n)] > 0)
    return mask * (1.0 - rng.random((n, n)))


@pytest.mark.parametrize("n", [21, 25, 27])
def test_exact_call(pb, n):
    A = _matrix(n, 1)
    with pb.Engine(0) as eng:
        want = eng.exact_dense(A, variant=pb.PERM_KERNEL_DENSE_SDD)
        for variant in (0, pb.PERM_KERNEL_DENSE):
            eng.inject_wait_timeout(1)
            with pytest.raises(pb.PermError, match="staging.*timed out") as ei:
                eng.exact_dense(A, variant=variant)
            assert ei.value.status == pb.PERM_ETIMEOUT
            for _ in range(2):
                r = eng.exact_dense(A, variant=variant)
                tol = (r.rel_error_estimate + want.rel_error_estimate + 2 * U) * want.value
                assert abs(r.value - want.value) <= tol


def test_batch(pb):
    mats = [_matrix(n, 2) for n in (12, 25, 26)]
    with pb.Engine(0) as eng:
        want = [eng.exact_dense(A).value for A in mats]
        eng.inject_wait_timeout(1)
        bad = eng.batch(mats)
        good = eng.batch(mats)
        try:
            for _ in range(2):
                with pytest.raises(pb.PermError, match="staging.*timed out") as ei:
                    bad.run()
                assert ei.value.status == pb.PERM_ETIMEOUT
                values, _ = good.run()
                assert np.all(np.abs(values - want) <= 1e-10 * np.abs(want))
        finally:
            bad.free()
            good.free()
