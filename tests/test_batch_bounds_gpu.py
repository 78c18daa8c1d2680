"""Error bounds of a batch's values: those of the walk that made each value."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _matrix(n, d, seed, integers):
    rng = np.random.default_rng([n, seed])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    return mask * (1.0 if integers else 1.0 - rng.random((n, n)))


@pytest.mark.parametrize("n,d,integers", [(22, 0.5, True), (24, 0.3, True), (24, 0.5, True), (26, 0.4, True),
                                          (18, 0.5, True), (23, 0.5, False), (26, 0.5, False), (18, 0.6, False)])
def test_target_just_below_the_own_bound(pb, n, d, integers):
    """A value whose own bound misses the target by a little is not kept for
    the smaller bound of another walk: it is evaluated again, or checked."""
    A = _matrix(n, d, 3, integers)
    with pb.Engine(0) as eng:
        certified = pb.PERM_KERNEL_DENSE_INT_DD if integers else pb.PERM_KERNEL_DENSE_SDD
        want = eng.exact_dense(A, variant=certified)
        b = eng.batch([A] * 3)
        try:
            eng.set_rel_target(0.0)
            values, own, reruns, _ = b.run_ex()
            assert reruns == 0 and np.all(own > 0.0)
            # the bound is of (hi, lo); their sum is rounded once more
            assert np.all(np.abs(values - want.value) <= (own + want.rel_error_estimate + 2 * U) * abs(want.value))
            for part in (0.75, 0.9):
                target = float(own.min()) * part
                eng.set_rel_target(target)
                values, est, reruns, _ = b.run_ex()
                assert reruns == 3 and np.all(est <= target)
                assert np.all(np.abs(values - want.value) <= (est + want.rel_error_estimate + 2 * U) * abs(want.value))
                if integers:  # no cross-check there: the certified value
                    assert np.all(est < 1e-14), est
        finally:
            b.free()


def test_estimates_repeat_to_the_bit(pb):
    """Sums of |term| are added in a fixed order: the bound of a value, and
    with it whether it is evaluated again, does not change between runs."""
    mats = [_matrix(n, d, 5, integers) for n in (18, 22, 24, 25, 27) for d in (0.3, 0.5) for integers in (True, False)]
    with pb.Engine(0) as eng:
        eng.set_rel_target(0.0)
        b = eng.batch(mats)
        try:
            first = b.run_ex()
            for _ in range(20):
                values, est, _, _ = b.run_ex()
                assert np.array_equal(values, first[0]) and np.array_equal(est, first[1])
        finally:
            b.free()
        for A in mats:
            for variant in (0, pb.PERM_KERNEL_DENSE_SDD):
                got = {(r.hi, r.lo, r.abs_term_sum) for r in (eng.exact_dense(A, variant=variant) for _ in range(10))
                       if len(A) >= 25}
                assert len(got) <= 1, (A.shape, variant, got)
