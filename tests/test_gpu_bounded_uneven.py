"""Bounded products (no bounds pass, no binning) whose rows do not suit one
table size: many rows past the tables of the bound, and one long row among
short ones.  Results equal the oracle's bit for bit, in every flavour."""
import numpy as np
import pytest

import oracle as O
import sp3mm4amg_b200 as S

pytestmark = pytest.mark.gpu


def _rows(rng, M, N, n):
    """Rows of up to n[i] random distinct columns."""
    import scipy.sparse as sp
    row = np.repeat(np.arange(M), n)
    m = sp.csr_matrix((rng.uniform(-1, 1, len(row)), (row, rng.integers(0, N, len(row)))),
                      shape=(M, N))
    m.sum_duplicates()
    m.sort_indices()
    return S.CSR(m.indptr.astype(np.int64), m.indices.astype(np.int64), m.data, m.shape)


def _between(rng, M, N, lo, hi):
    return _rows(rng, M, N, rng.integers(lo, hi + 1, M))


def _labels(orc, ops, vt=S.F64):
    """{flavour: labels} of the product, checked against the oracle (FP64) or
    the binned path (FP32; lane tuning takes it)."""
    out = {}
    with S.Context() as ctx:
        d = [ctx.upload(m, vt) for m in ops]
        run = (lambda fl: ctx.rap(*d, S.DIRECT, fl, vt)) if len(d) == 3 else \
            (lambda fl: ctx.spmm(*d, fl, vt))
        for fl in (S.UB, S.SYMBNUM):
            ctx.set_profiling(True)
            C = run(fl)
            out[fl] = set(ctx.profile())
            ctx.set_profiling(False)
            got = C.download()
            C.free()
            if vt == S.F64:
                want = orc.spmm(*ops) if len(ops) == 2 else orc.sp3mm_direct(*ops)
                cmp = O.compare(got, want, rtol=0.0)
                assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (fl, cmp)
            else:
                ctx.set_tuning(32)
                C = run(fl)
                want = C.download()
                C.free()
                ctx.set_tuning(0)
                assert np.array_equal(got.indptr, want.indptr)
                assert np.array_equal(got.indices, want.indices)
                assert np.array_equal(got.data, want.data)
        for m in d:
            m.free()
    return out


@pytest.mark.parametrize("vt", [S.F64, S.F32])
@pytest.mark.parametrize("M", [7000, 20000])
def test_rows_past_the_tables_are_binned_by_their_counts(orc, M, vt):
    # With and without the replayed kernel's try; empty rows among them.
    rng = np.random.default_rng(M)
    ops = [_between(rng, M, M, 0, 6), _between(rng, M, M, 5, 15), _between(rng, M, M // 2, 1, 3)]
    labels = _labels(orc, ops, vt)
    assert "bin.levels" in labels[S.SYMBNUM], labels
    assert "bin.levels" not in labels[S.UB], labels
    assert ("direct.replay.symb" in labels[S.SYMBNUM]) == (M >= 16384), labels


def test_few_rows_past_the_tables_are_not(orc):
    from sp3mm4amg_b200 import problems as pb
    p = pb.stencil_problem(3, (50, 48, 52))
    labels = _labels(orc, [p.R, p.A, p.P])
    assert "bin.levels" not in labels[S.SYMBNUM], labels


@pytest.mark.parametrize("M,longest,binned", [(149999, 60, False), (150000, 60, True),
                                              (150000, 24, False)])
def test_one_long_row_among_many_short(orc, M, longest, binned):
    # From 150,000 rows on, rows far past the mean (32 times its products) take
    # the whole product to the bounds and the bins.
    rng = np.random.default_rng(longest)
    n = rng.integers(1, 4, M)
    n[M // 3] = longest
    A, B = _rows(rng, M, 5000, n), _between(rng, 5000, 5000, 2, 8)
    for ops in ([A, B], [A, B, _between(rng, 5000, 3000, 1, 3)]):
        for fl, labels in _labels(orc, ops).items():
            assert any(x.endswith(".bounds") for x in labels) == binned, (fl, labels)
