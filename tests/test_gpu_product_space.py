"""Booked space of the upper-bound flavour: products whose space is enough are
formed in one pass (no symbolic pass follows), replayed rows included; where it
is not, results are the same."""
import numpy as np
import pytest

import oracle as O
import sp3mm4amg_b200 as S

pytestmark = pytest.mark.gpu


def _passes(ctx, f):
    """f()'s result and the labels of the passes that it ran."""
    ctx.set_profiling(True)
    C = f()
    labels = set(ctx.profile())
    ctx.set_profiling(False)
    return C, labels


def _booked_once(labels):
    return any(x.endswith(".book") for x in labels) and \
        not any(x.endswith((".symb", ".num")) for x in labels)


def _same(C, want, what):
    cmp = O.compare(C.download(), want, rtol=0.0)
    assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (what, cmp)


def _ladder(rng, M, k, l):
    """A (k entries a row) and B (l a row) whose product's rows hold k*l
    columns, each row's shifted by l from the one before."""
    A = S.CSR(np.arange(M + 1, dtype=np.int64) * k,
              (np.arange(M, dtype=np.int64)[:, None] + np.arange(k)).ravel(),
              rng.uniform(-1, 1, M * k), (M, M + k - 1))
    n = M + k - 1
    B = S.CSR(np.arange(n + 1, dtype=np.int64) * l, np.arange(n * l, dtype=np.int64),
              rng.uniform(-1, 1, n * l), (n, n * l))
    return A, B


def test_replayed_rows_fill_their_space(orc):
    # Every product is a column, so the space is exactly the result's entries
    # and the warps' last handouts; rows of 86 do not divide a handout.
    A, B = _ladder(np.random.default_rng(1), 200000, 2, 43)
    want = orc.spmm(A, B)
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in (A, B)]
        for fl in (S.UB, S.SYMBNUM):
            C, labels = _passes(ctx, lambda: ctx.spmm(*d, fl))
            assert any(x.startswith("pair.replay") for x in labels)
            assert _booked_once(labels) == (fl == S.UB), labels
            _same(C, want, fl)
            C.free()
        for m in d:
            m.free()


def test_batch_overflows_after_replayed_rows(orc):
    # 60,000 rows of 64 columns each, most of them shifted copies of one
    # pattern (replayed), some not; far more entries than twice the operands'
    # and the handouts, so the batch is planned again symbolically.  A second
    # run with new values replays the numeric pass.
    rng = np.random.default_rng(2)
    cols = [np.arange(64) * 3 + i for i in range(40)]
    cols += [np.sort(rng.choice(320, 64, replace=False)) for _ in range(4)]
    A = S.CSR(np.arange(45, dtype=np.int64) * 64, np.concatenate(cols).astype(np.int64),
              rng.uniform(-1, 1, 44 * 64), (44, 320))
    P = S.CSR(np.arange(321, dtype=np.int64), np.arange(320, dtype=np.int64),
              rng.uniform(-1, 1, 320), (320, 320))
    M = 60000
    pick = np.where(rng.random(M) < 0.02, rng.integers(40, 44, M), rng.integers(0, 40, M))
    Rs = [S.CSR(np.arange(M + 1, dtype=np.int64), pick[rng.permutation(M)].astype(np.int64),
                rng.uniform(-1, 1, M), (M, 44)) for _ in range(2)]
    with S.Context() as ctx:
        d = [[ctx.upload(m) for m in (R, A, P)] for R in Rs]
        b = ctx.batch([tuple(x) for x in d], S.F64, S.UB)
        ctx.set_profiling(True)
        b.run()
        labels = set(ctx.profile())
        ctx.set_profiling(False)
        assert "batch.replay" in labels and "batch.symbolic" in labels, labels
        for step in range(2):
            for i, R in enumerate(Rs):
                _same(b.result(i), orc.sp3mm_direct(R, A, P), (step, i))
            A = S.CSR(A.indptr, A.indices, rng.uniform(-1, 1, A.nnz), A.shape)
            for x in d:
                x[1].set_values(A.data)
            b.run()
        b.free()
        for x in d:
            for m in x:
                m.free()
