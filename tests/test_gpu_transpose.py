"""Transpose (column counts, scan, scatter, row sort): rows of the transpose
on both sides of the sort's switches (32 and 2048 entries), both value types,
the longest row, and a column that a row holds twice, which is refused."""
import numpy as np
import pytest

import sp3mm4amg_b200 as S

pytestmark = pytest.mark.gpu


def _tall(lengths, N, seed):
    """A CSR whose column c holds lengths[c] entries at random rows."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.choice(N, n, replace=False) for n in lengths] + [[]]).astype(int)
    cols = np.repeat(np.arange(len(lengths)), lengths)
    order = np.lexsort((cols, rows))
    ptr = np.zeros(N + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=N), out=ptr[1:])
    return S.CSR(ptr, cols[order].astype(np.int64), rng.uniform(-1, 1, len(cols)),
                 (N, len(lengths)))


@pytest.mark.parametrize("vt", [S.F64, S.F32])
@pytest.mark.parametrize("lengths", [
    [0, 1, 2, 31, 32, 33, 34, 0, 127, 128, 129, 511, 513, 2047, 2048, 2049, 2500, 5],
    [1], [0, 0], list(range(40)) * 3])
def test_row_lengths(lengths, vt):
    A = _tall(lengths, 2600, len(lengths))
    if vt == S.F32:
        A.data[:] = A.data.astype(np.float32)
    want = A.transpose()
    with S.Context() as ctx:
        dA = ctx.upload(A, vt)
        dT = ctx.transpose(dA)
        got = dT.download()
        assert dT.max_row == (max(lengths) if lengths else 0)
        dT.free()
        dA.free()
    assert np.array_equal(got.indptr, want.indptr)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.data, want.data)


@pytest.mark.parametrize("n", [3, 40, 2100])
def test_repeated_column_is_refused(n):
    # Upload refuses such a row, so the device copy's columns are overwritten.
    import torch
    A = _tall([n, n], n + 5, 7)
    with S.Context() as ctx:
        dA = ctx.upload(A)
        row = int(np.argmax(np.diff(A.indptr)))    # a row of both columns
        assert A.indptr[row + 1] - A.indptr[row] == 2

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
