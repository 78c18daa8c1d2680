"""Row-layout walks at the orders where whole calls take column cubes
(perm_exact_dense_rows): every family of layouts that densities 0.12..0.8 lead
to (two and three levels of FP64 x, split-dd, int32 x and certified int32 x),
whole and in shards, against the certified column-cube walk within the sum of
both bounds; and the completion of a checkpoint that was begun in rows."""
from __future__ import annotations

import json

import numpy as np
import pytest

U = 2.0 ** -53


def _matrix(n, d, seed, integers):
    rng = np.random.default_rng([n, seed])
    mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
    return mask * (rng.integers(1, 5, (n, n)).astype(np.float64) if integers else 1.0 - rng.random((n, n)))


def _families(pb, A, integers):
    if integers:
        _, ngo, ng1, _ = pb.int_layout(A)
        _, pair, cgo, cg1, _ = pb.intc_layout(A)
        return {("int", bool(ngo), bool(ng1)), ("intc", pair, bool(cgo), bool(cg1))}
    return {("fp64",) + pb.fp64_levels(A), ("sdd",) + pb.sdd_levels(A)}


@pytest.mark.gpu
@pytest.mark.parametrize("n,integers", [(25, False), (27, False), (28, False), (30, False), (33, False), (25, True),
                                        (27, True), (28, True), (30, True), (33, True)])
def test_row_layouts_vs_certified_cubes(engine, pb, n, integers):
    plain, certified = ((pb.PERM_KERNEL_DENSE_INT, pb.PERM_KERNEL_DENSE_INT_DD) if integers
                        else (pb.PERM_KERNEL_DENSE, pb.PERM_KERNEL_DENSE_SDD))
    seen = set()
    for d in (0.12, 0.2, 0.3, 0.4, 0.5, 0.6, 0.7, 0.8):
        for seed in range(3 if n < 33 else 1):
            A = _matrix(n, d, seed, integers)
            seen |= _families(pb, A, integers)
            want = engine.exact_dense(A, variant=certified)
            for variant in (plain, certified):
                r = engine.exact_dense_rows(A, variant=variant)
                assert r.kernel == variant and r.steps == r.total_steps
                tol = (r.rel_error_estimate + want.rel_error_estimate + 2 * U) * abs(want.value)
                assert abs(r.value - want.value) <= tol, (d, seed, variant, r.value, want.value, tol)
                if seed == 0:
                    parts = [engine.exact_dense_rows(A, s, 3, variant=variant) for s in range(3)]
                    hi, lo = pb.dd_sum([(p.hi, p.lo) for p in parts])
                    assert abs(hi + lo - want.value) <= 2 * tol, (d, variant)
    levels = {f[:1] + tuple(bool(x) for x in f[-2:]) for f in seen}
    kinds = ("int", "intc") if integers else ("fp64", "sdd")
    three = (False, True) if integers else (True, True)
    for kind in kinds:
        if n >= 28 or kind == "sdd":
            assert (kind,) + three in levels, levels
        if n < 28:
            assert (kind,) + ((True, False) if integers else (False, True)) in levels, levels


class _Engine:
    """Shards of a known sum from two walks that must not be mixed."""

    def __init__(self):
        self.calls = []

    def _part(self, kind, shard):
        from types import SimpleNamespace

        self.calls.append((kind, shard))
        return SimpleNamespace(hi=float((1 if kind == "rows" else 100) * (shard + 1)), lo=0.0)

    def exact_dense_rows(self, mat, shard=0, nshards=1, variant=0):
        return self._part("rows", shard)

    def exact_dense_shard(self, mat, shard, nshards, variant=0):
        return self._part("shard", shard)


def _write(pb, path, A, fmt, variant, done):
    a = np.ascontiguousarray(A)
    path.write_text(json.dumps({"format": fmt, "matrix_sha256": pb._fingerprint(a), "n": len(a), "chunks": 4,
                                "variant": variant, "done": {str(c): [float(h).hex(), 0.0.hex()] for c, h in done}}))


def test_checkpoint_begun_in_rows_is_completed_in_rows(pb, tmp_path):
    A = _matrix(26, 0.5, 0, False)
    path = tmp_path / "walk.ckpt"
    _write(pb, path, A, "perm_b200_checkpoint_v1", 0, [(0, 1.0), (2, 3.0)])
    eng = _Engine()
    assert pb.checkpointed_exact_dense(A, path, chunks=4, engine=eng, keep=True) == (10.0, 0.0)
    assert eng.calls == [("rows", 1), ("rows", 3)]
    # still a file of that walk
    assert json.loads(path.read_text())["format"] == "perm_b200_checkpoint_v1"
    assert pb.checkpointed_exact_dense(A, path, chunks=4, engine=eng) == (10.0, 0.0) and len(eng.calls) == 2
    # a new walk takes the cubes, an order below them walks rows by itself
    assert pb.checkpointed_exact_dense(A, path, chunks=4, engine=eng) == (1000.0, 0.0)
    pb.checkpointed_exact_dense(A[:24, :24], path, chunks=4, engine=eng)
    assert [k for k, _ in eng.calls[2:]] == ["shard"] * 8
    # whoever brings the shards' walk has to bring the file's
    _write(pb, path, A, "perm_b200_checkpoint_v1", 0, [(0, 1.0)])
    with pytest.raises(pb.PermError, match="format"):
        pb.checkpointed_exact_dense(A, path, chunks=4, shard_fn=lambda m, c, k: (1.0, 0.0))


def test_checkpoint_of_an_unknown_side_is_refused(pb, tmp_path):
    """Certified walks of the format before may have walked the transpose."""
    A = _matrix(26, 0.5, 0, False)
    path = tmp_path / "walk.ckpt"
    for variant, ok in ((0, True), (pb.PERM_KERNEL_DENSE, True), (pb.PERM_KERNEL_DENSE_INT_DD, False),
                        (pb.PERM_KERNEL_DENSE_SDD, False)):
        _write(pb, path, A, "perm_b200_checkpoint_v2", variant, [(0, 100.0), (1, 200.0)])
        if ok:
            assert pb.checkpointed_exact_dense(A, path, chunks=4, variant=variant, engine=_Engine()) == (1000.0, 0.0)
        else:
            with pytest.raises(pb.PermError, match="format"):
                pb.checkpointed_exact_dense(A, path, chunks=4, variant=variant, engine=_Engine())


@pytest.mark.gpu
def test_checkpoint_begun_in_rows_on_the_gpu(pb, engine, tmp_path):
    A = _matrix(27, 0.5, 1, False)
    for variant in (0, pb.PERM_KERNEL_DENSE_SDD):
        path = tmp_path / f"walk{variant}.ckpt"
        first = [(c, engine.exact_dense_rows(A, c, 4, variant=variant)) for c in (0, 3)]
        path.write_text(json.dumps({"format": "perm_b200_checkpoint_v1", "matrix_sha256": pb._fingerprint(A), "n": 27,
                                    "chunks": 4, "variant": variant,
                                    "done": {str(c): [p.hi.hex(), p.lo.hex()] for c, p in first}}))
        hi, lo = pb.checkpointed_exact_dense(A, path, chunks=4, variant=variant, engine=engine)
        want = engine.exact_dense(A)
        bound = engine.exact_dense_rows(A, variant=variant or pb.PERM_KERNEL_DENSE).rel_error_estimate
        assert abs(hi + lo - want.value) <= (bound + want.rel_error_estimate + 2 * U) * abs(want.value)


@pytest.mark.gpu
@pytest.mark.parametrize("n,top,variant", [(25, 4, "PERM_KERNEL_DENSE_INT"), (27, 4, "PERM_KERNEL_DENSE_INT"),
                                           (28, 4, "PERM_KERNEL_DENSE_INT"), (25, 0, "PERM_KERNEL_DENSE")])
def test_cubes_are_as_exact_as_rows(engine, pb, n, top, variant):
    """Errors of one plain walk against the certified value, in units of
    sum |term|: over 300 matrices the cubes' rms is no larger than the row
    layouts' (top 0: FP32 values, whose x are exact too)."""
    variant = getattr(pb, variant)
    certified = pb.PERM_KERNEL_DENSE_INT_DD if top else pb.PERM_KERNEL_DENSE_SDD
    square = np.zeros(2)
    engine.set_rel_target(0.0)
    try:
        for d in (0.35, 0.5, 0.7):
            for seed in range(100):
                rng = np.random.default_rng([n, seed, 77])
                mask = (rng.random((n, n)) < d) | (np.eye(n)[rng.permutation(n)] > 0)
                A = mask * (rng.integers(1, top + 1, (n, n)) if top else np.float32(1.0 - rng.random((n, n))))
                A = A.astype(np.float64)
                c = engine.exact_dense(A, variant=certified)
                for k, r in enumerate((engine.exact_dense_shard(A, 0, 1, variant=variant),
                                       engine.exact_dense_rows(A, variant=variant))):
                    square[k] += (((r.hi - c.hi) + (r.lo - c.lo)) / (U * c.abs_term_sum)) ** 2
    finally:
        engine.set_rel_target(1e-10)
    assert square[0] <= square[1], np.sqrt(square / 300)
