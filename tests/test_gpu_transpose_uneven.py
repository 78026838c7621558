"""Transposes of matrices whose rows differ widely in length: the same result,
and one long row among short ones takes about what the long row and the short
ones take apart."""
import time

import numpy as np
import pytest

import sp3mm4amg_b200 as S

pytestmark = pytest.mark.gpu


def _rows(rng, lengths, N):
    """Rows of the given numbers of distinct columns, ascending."""
    cols = [np.sort(rng.choice(N, n, replace=False)) if n > 8 else
            np.unique(rng.integers(0, N, n)) for n in lengths]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    return S.CSR(ptr, np.concatenate(cols).astype(np.int64), rng.uniform(-1, 1, int(ptr[-1])),
                 (len(lengths), N))


def _times(ctx, A):
    d = ctx.upload(A)
    t = []
    for _ in range(8):
        ctx.sync()
        t0 = time.perf_counter()
        ctx.transpose(d).free()
        ctx.sync()
        t.append(time.perf_counter() - t0)
    d.free()
    return min(t)


@pytest.mark.parametrize("mean", [1, 3, 9, 20])
def test_long_rows_among_short(mean):
    # Every number of lanes per row, rows at their limit (8 times the lanes)
    # and beyond it, several in one warp, the last row among them.
    rng = np.random.default_rng(mean)
    n = rng.integers(0, 2 * mean + 1, 3001)
    lanes = 1 << int(np.ceil(np.log2(mean)))
    n[[3, 4, 5, 700, 3000]] = [8 * lanes, 8 * lanes + 1, 8 * lanes - 1, 1900, 1500]
    A = _rows(rng, n, 2000)
    want = A.transpose()
    with S.Context() as ctx:
        d = ctx.upload(A)
        T = ctx.transpose(d)
        got = T.download()
        T.free()
        d.free()
    assert np.array_equal(got.indptr, want.indptr)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.data, want.data)


def test_one_long_row_costs_no_more_than_alone():
    rng = np.random.default_rng(5)
    short = np.full(200000, 2)
    both = short.copy()
    both[777] = 150000
    with S.Context() as ctx:
        t_short = _times(ctx, _rows(rng, short, 200000))
        t_long = _times(ctx, _rows(rng, [150000], 200000))
        t_both = _times(ctx, _rows(rng, both, 200000))
    # (on the lanes of its neighbours the long row took six times as long)
    assert t_both < 2 * (t_short + t_long), (t_short, t_long, t_both)


@pytest.mark.parametrize("vt", [S.F64, S.F32])
def test_rows_on_both_sides_of_the_network(vt):
    rng = np.random.default_rng(6)
    T = _rows(rng, [1023, 1024, 1025, 1026, 1500, 2046, 2047, 2048, 1025], 5000)
    if vt == S.F32:
        T.data[:] = T.data.astype(np.float32)
    with S.Context() as ctx:
        d = ctx.upload(T.transpose(), vt)
        got = ctx.transpose(d).download()
        d.free()
    assert np.array_equal(got.indptr, T.indptr)
    assert np.array_equal(got.indices, T.indices)
    assert np.array_equal(got.data, T.data)


@pytest.mark.parametrize("n", [1025, 2048])
def test_repeated_column_is_refused(n):
    # Upload refuses such a row, so the device copy's columns are overwritten.
    import torch
    A = _rows(np.random.default_rng(7), [n, n], n + 5).transpose()
    with S.Context() as ctx:
        dA = ctx.upload(A)
        row = int(np.argmax(np.diff(A.indptr)))    # a row of both columns

        class Mem:
            __cuda_array_interface__ = {"shape": (A.nnz,), "typestr": "<i4",
                                        "data": (dA.d.col, False), "version": 3}
        cols = torch.as_tensor(Mem(), device="cuda")
        ctx.sync()
        cols[int(A.indptr[row]) + 1] = 0           # column 0 twice in one row
        torch.cuda.synchronize()
        with pytest.raises(S.Sp3mmError):
            ctx.transpose(dA)
        dA.free()


def test_time_does_not_grow_with_the_rows_length():
    # As many entries in rows of 2,000 as in rows of 1,000 (ranks alone: 1.6
    # times as long).
    rng = np.random.default_rng(8)
    t = {}
    with S.Context() as ctx:
        for n in (1000, 2000):
            A = _rows(rng, [n] * (2000000 // n), 16 * n).transpose()
            t[n] = _times(ctx, A)
    assert t[2000] < 1.2 * t[1000], t
