"""Infinities, NaN, signed zeros and subnormals through the kernels of bounded
products (a thread per row, replayed rows, the lanes kernel), single and in a
batch: patterns depend on columns only, and values come out as the oracle's;
and a planned batch whose operand's columns have changed, which is reported."""
import numpy as np
import pytest

import sp3mm4amg_b200 as S
from sp3mm4amg_b200 import problems as pb

pytestmark = pytest.mark.gpu

SPECIAL = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 5e-324, -1e-310, 1e308, -1e308])


def _special(m, rng, share):
    v = rng.uniform(-1, 1, m.nnz)
    at = rng.random(m.nnz) < share
    v[at] = rng.choice(SPECIAL, int(at.sum()))
    return S.CSR(m.indptr, m.indices, v, m.shape)


def _same(got, want, what):
    assert np.array_equal(got.indptr, want.indptr), what
    assert np.array_equal(got.indices, want.indices), what
    a, b = np.asarray(got.data), np.asarray(want.data)
    assert np.array_equal(np.isnan(a), np.isnan(b)), what
    ok = ~np.isnan(a)
    assert np.array_equal(a[ok].view(np.int64), b[ok].view(np.int64)), what


@pytest.mark.parametrize("dims", [(290, 281), (57, 55, 53), (40, 37)])
@pytest.mark.parametrize("variant", [S.DIRECT, S.PAIR, S.PAIR_RIGHT])
def test_single_products(orc, dims, variant):
    rng = np.random.default_rng(sum(dims))
    p = pb.stencil_problem(len(dims), dims)
    with np.errstate(all="ignore"):
        ops = [_special(m, rng, 0.002) for m in (p.R, p.A, p.P)]
        want = {S.DIRECT: orc.sp3mm_direct, S.PAIR: orc.sp3mm_pair,
                S.PAIR_RIGHT: orc.sp3mm_pair_right}[variant](*ops)
    assert np.isnan(want.data).any() and np.isfinite(want.data).any()
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in ops]
        for fl in (S.UB, S.SYMBNUM):
            C = ctx.rap(*d, variant, fl)
            _same(C.download(), want, (dims, variant, fl))
            C.free()
        for m in d:
            m.free()


def _batch(ctx, rng, fl):
    p = pb.stencil_problem(2, (300, 260))
    ops = [_special(m, rng, 0.002) for m in (p.R, p.A, p.P)]
    d = [ctx.upload(m) for m in ops]
    return ops, d, ctx.batch([tuple(d)], S.F64, fl)


@pytest.mark.parametrize("fl", [S.UB, S.SYMBNUM])
def test_batches(orc, fl):
    rng = np.random.default_rng(3)
    with S.Context() as ctx:
        ops, d, b = _batch(ctx, rng, fl)
        b.run()
        _same(b.result(0).download(), orc.sp3mm_direct(*ops), fl)
        b.execute()                       # the replayed numeric pass
        _same(b.result(0).download(), orc.sp3mm_direct(*ops), fl)
        b.free()
        for m in d:
            m.free()


def test_changed_columns_of_a_planned_batch_are_reported():
    # One entry moved to a free column of its row, in range: a replayed row
    # whose products no longer lie as the template's.
    import torch
    rng = np.random.default_rng(4)
    with S.Context() as ctx:
        ops, d, b = _batch(ctx, rng, S.UB)
        b.run()
        b.execute()
        ctx.sync()

        class Mem:
            __cuda_array_interface__ = {"shape": (ops[1].nnz,), "typestr": "<i4",
                                        "data": (d[1].d.col, False), "version": 3}
        cols = torch.as_tensor(Mem(), device="cuda")
        row = 130 * 300 + 150             # inside: columns row - 300, row - 1, row, ...
        at = int(ops[1].indptr[row])
        cols[at] = row - 2 * 300
        torch.cuda.synchronize()
        with pytest.raises(S.Sp3mmError):
            b.execute()
            b.result(0).download()
            ctx.transpose(d[0])           # (the next call that reads the error word)
        cols[at] = row - 300
        torch.cuda.synchronize()
        b.execute()
        ctx.sync()
        b.free()
        for m in d:
            m.free()
