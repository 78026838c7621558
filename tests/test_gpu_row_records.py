"""A caller's sp3mm_dcsr that records too short a longest row (or none): SpMM,
its row sizes and the direct product's left operand do not depend on it."""
import numpy as np
import pytest

import oracle as O
import sp3mm4amg_b200 as S

pytestmark = pytest.mark.gpu


def _rows(rng, M, N, lo, hi):
    import scipy.sparse as sp
    row = np.repeat(np.arange(M), rng.integers(lo, hi + 1, M))
    m = sp.csr_matrix((rng.uniform(-1, 1, len(row)), (row, rng.integers(0, N, len(row)))),
                      shape=(M, N))
    m.sum_duplicates()
    m.sort_indices()
    return S.CSR(m.indptr.astype(np.int64), m.indices.astype(np.int64), m.data, m.shape)


def _same(C, want, what):
    cmp = O.compare(C.download(), want, rtol=0.0)
    assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (what, cmp)
    C.free()


# name: (M, entries of A's rows, of B's rows): a thread per row, the lanes
# kernel, the replayed kernel's try, and rows past the bounded path.
SIZES = {"tiny": (500, 6, 5), "lanes": (700, 16, 16), "replay": (17000, 16, 12),
         "binned": (300, 40, 40)}


@pytest.mark.parametrize("size", list(SIZES))
@pytest.mark.parametrize("said", [0, 1, 2, -1])
@pytest.mark.parametrize("which", ["A", "B", "both"])
def test_spmm(orc, size, said, which):
    M, a, b = SIZES[size]
    rng = np.random.default_rng(M)
    A, B = _rows(rng, M, 400, 0, a), _rows(rng, 400, 900, b // 2, b)
    want = orc.spmm(A, B)
    with S.Context() as ctx:
        dA, dB = ctx.upload(A), ctx.upload(B)
        if which != "B":
            dA.d.max_row = said
        if which != "A":
            dB.d.max_row = said
        for fl in (S.UB, S.SYMBNUM):
            _same(ctx.spmm(dA, dB, fl), want, (size, said, which, fl))
        rows, total = ctx.rowsizes(dA, dB)
        assert total == want.nnz and np.array_equal(rows, np.diff(want.indptr))
        dA.free()
        dB.free()


@pytest.mark.parametrize("M", [600, 17000])
@pytest.mark.parametrize("said", [0, 1, 3, -1])
def test_direct(orc, M, said):
    rng = np.random.default_rng(M + said)
    ops = [_rows(rng, M, 400, 0, 12), _rows(rng, 400, 900, 8, 16), _rows(rng, 900, 300, 1, 4)]
    want = orc.sp3mm_direct(*ops)
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in ops]
        d[0].d.max_row = said
        for fl in (S.UB, S.SYMBNUM):
            _same(ctx.rap(*d, S.DIRECT, fl), want, (M, said, fl))
        for m in d:
            m.free()
