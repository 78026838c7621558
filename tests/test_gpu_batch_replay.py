"""Which rows of a batch the numeric pass replays: runs of rows that the plan's
pass mostly replayed, the others on the tiers, in both flavours; results equal
the oracle's bit for bit, also after new values."""
import numpy as np
import pytest

import oracle as O
import sp3mm4amg_b200 as S
from sp3mm4amg_b200 import problems as pb

pytestmark = pytest.mark.gpu


def _random(rng, M, N, lo, hi):
    import scipy.sparse as sp
    row = np.repeat(np.arange(M), rng.integers(lo, hi + 1, M))
    m = sp.csr_matrix((rng.uniform(-1, 1, len(row)), (row, rng.integers(0, N, len(row)))),
                      shape=(M, N))
    m.sum_duplicates()
    m.sort_indices()
    return S.CSR(m.indptr.astype(np.int64), m.indices.astype(np.int64), m.data, m.shape)


def _irregular(rng, M):
    return [_random(rng, M, M, 3, 6), _random(rng, M, M, 5, 15), _random(rng, M, M // 2, 1, 3)]


def _grid(dims, rng, broken=0.0):
    p = pb.stencil_problem(len(dims), dims)
    m = p.A.to_scipy().copy()
    m.data[:] = rng.uniform(-1, 1, m.nnz)
    m.data[rng.random(m.nnz) < broken] = 0.0
    m.eliminate_zeros()
    return [p.R, S.CSR.from_scipy(m), p.P]


# name: (products, how many classes of rows are replayed)
BATCHES = {
    "irregular": (lambda r: [_irregular(r, M) for M in (5000, 16000, 3000)], 0),
    "grids": (lambda r: [_grid(d, r) for d in ((300, 260), (60, 50, 55))], 2),
    # about a third of the rows of the broken grids match
    "partly": (lambda r: [_grid((300, 260), r, 0.03), _grid((60, 50, 55), r, 0.01)], None),
    "mixed": (lambda r: [_grid((300, 260), r), _irregular(r, 9000), _grid((250, 240), r, 0.03)], 1),
}


@pytest.mark.parametrize("fl", [S.UB, S.SYMBNUM])
@pytest.mark.parametrize("which", list(BATCHES))
def test_rows_replayed_in_the_numeric_pass(orc, which, fl):
    rng = np.random.default_rng(len(which))
    make, classes = BATCHES[which]
    ops = make(rng)
    with S.Context() as ctx:
        d = [[ctx.upload(m) for m in o] for o in ops]
        b = ctx.batch([tuple(x) for x in d], S.F64, fl)
        b.run()
        for step in range(2):
            for i, o in enumerate(ops):
                want = orc.sp3mm_direct(*o)
                cmp = O.compare(b.result(i).download(), want, rtol=0.0)
                assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (which, step, i, cmp)
            for o, x in zip(ops, d):
                o[1] = S.CSR(o[1].indptr, o[1].indices, rng.uniform(-1, 1, o[1].nnz), o[1].shape)
                x[1].set_values(o[1].data)
            b.execute()
        # Other table sizes capture the numeric pass again: its launches.
        before = ctx.launches()
        b.set_tuning(slack=1)
        replays = ctx.launches() - before - b.info()["tiers"]
        assert classes is None or replays == classes, (which, replays)
        b.execute()
        for i, o in enumerate(ops):
            want = orc.sp3mm_direct(*o)
            cmp = O.compare(b.result(i).download(), want, rtol=0.0)
            assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (which, i, cmp)
        b.free()
        for x in d:
            for m in x:
                m.free()


@pytest.mark.parametrize("fl", [S.UB, S.SYMBNUM])
@pytest.mark.parametrize("rows", [4096, 4097])
def test_small_rows_in_one_tier(orc, rows, fl):
    # Rows of 0 to 100 products on both sides of the count up to which the
    # plan's pass gives them one launch, with heavier rows beside them.
    rng = np.random.default_rng(rows)
    A, P = _random(rng, 500, 700, 1, 10), _random(rng, 700, 300, 1, 3)
    ops = [[_random(rng, rows - 300, 500, 0, 10), A, P], [_random(rng, 300, 500, 1, 3), A, P],
           [_random(rng, 200, 500, 60, 90), A, P]]
    pair = (ops[0][0], A)
    with S.Context() as ctx:
        d = [[ctx.upload(m) for m in o] for o in ops + [list(pair)]]
        b = ctx.batch([tuple(x) for x in d], S.F64, fl)
        b.run()
        for i, want in enumerate([orc.sp3mm_direct(*o) for o in ops] + [orc.spmm(*pair)]):
            cmp = O.compare(b.result(i).download(), want, rtol=0.0)
            assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (i, cmp)
        b.free()
        for x in d:
            for m in x:
                m.free()
