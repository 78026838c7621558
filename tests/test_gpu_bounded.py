"""Products whose longest rows bound every row's products (no bounds pass, no
binning): the replayed rows (rowreplay.cuh), the lanes kernels over all rows
or over what the replay leaves, and the thread-per-row SpMM (rowtiny.cuh).
Results must be bit-identical to the oracle and to the binned path (lane
tuning takes it), in every flavour and value type."""
import numpy as np
import pytest

import oracle as O
import sp3mm4amg_b200 as S
from sp3mm4amg_b200 import problems as pb

pytestmark = pytest.mark.gpu


def _equal(got, want, what):
    assert np.array_equal(got.indptr, want.indptr), what
    assert np.array_equal(got.indices, want.indices), what
    assert np.array_equal(np.asarray(got.data).view(np.int64),
                          np.asarray(want.data).view(np.int64)), what


def _run(ctx, ops, variant, fl, vt, lanes):
    d = [ctx.upload(m, val_type=vt) for m in ops]
    ctx.set_tuning(lanes)
    C = ctx.rap(*d, variant, fl, vt) if len(d) == 3 else ctx.spmm(*d, fl, vt)
    out = C.download()
    ctx.set_tuning(0)
    for m in [C] + d:
        m.free()
    return out


def _check(orc, ops, variant=S.DIRECT, what=""):
    want = (orc.spmm(*ops) if len(ops) == 2 else
            orc.sp3mm_direct(*ops) if variant == S.DIRECT else
            orc.sp3mm_pair(*ops) if variant == S.PAIR else orc.sp3mm_pair_right(*ops))
    with S.Context() as ctx:
        for fl in (S.UB, S.SYMBNUM):
            got = _run(ctx, ops, variant, fl, S.F64, 0)
            cmp = O.compare(got, want, rtol=0.0)
            assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (what, fl, cmp)
            _equal(_run(ctx, ops, variant, fl, S.F32, 0), _run(ctx, ops, variant, fl, S.F32, 32),
                   (what, fl, "f32"))


def _rows(rng, M, N, lo, hi):
    """Rows of lo to hi random distinct columns, random values."""
    n = rng.integers(lo, hi + 1, M)
    cols = [np.sort(rng.choice(N, k, replace=False)) for k in n]
    ptr = np.zeros(M + 1, np.int64)
    np.cumsum(n, out=ptr[1:])
    ci = np.concatenate(cols).astype(np.int64) if ptr[-1] else np.zeros(0, np.int64)
    return S.CSR(ptr, ci, rng.uniform(-1, 1, int(ptr[-1])), (M, N))


def _random_values(m, rng):
    return S.CSR(m.indptr, m.indices, rng.uniform(-1, 1, m.nnz), m.shape)


@pytest.mark.parametrize("dims", [(57, 55, 53), (300, 281)])
@pytest.mark.parametrize("variant", [S.DIRECT, S.PAIR, S.PAIR_RIGHT])
def test_stencils(orc, dims, variant):
    # At least 16,384 rows (coarse for the direct product), odd edges.
    rng = np.random.default_rng(1)
    p = pb.stencil_problem(len(dims), dims)
    _check(orc, [_random_values(m, rng) for m in (p.R, p.A, p.P)], variant, dims)


@pytest.mark.parametrize("which", ["A", "P"])
def test_broken_patterns(orc, which):
    # Entries of A (both stages differ) or of P alone (stage 2 differs) taken
    # out at random: rows that match the template in part.
    rng = np.random.default_rng(2)
    p = pb.stencil_problem(2, (290, 262))
    ops = {"R": p.R, "A": p.A, "P": p.P}
    m = ops[which].to_scipy().copy()
    m.data[rng.random(m.nnz) < 0.01] = 0.0
    m.eliminate_zeros()
    ops[which] = S.CSR.from_scipy(m)
    _check(orc, list(ops.values()), what=which)


def test_same_lengths_other_columns(orc):
    # Constant row lengths with random columns: only the column check tells
    # the rows apart.
    rng = np.random.default_rng(3)
    R = _rows(rng, 16500, 900, 4, 4)
    A = _rows(rng, 900, 800, 12, 12)
    P = _rows(rng, 800, 700, 3, 3)
    _check(orc, [R, A, P])
    _check(orc, [R, A], what="pair")


def test_rows_past_the_capacities(orc):
    # 200 distinct columns of 200 products: more than the template holds, and
    # more than the lanes kernel's first tables (retried rows); empty rows.
    rng = np.random.default_rng(4)
    R = _rows(rng, 16400, 60, 0, 2)
    A = _rows(rng, 60, 4000, 90, 100)
    P = _rows(rng, 4000, 3000, 0, 3)
    _check(orc, [R, A, P])
    _check(orc, [R, A], what="pair")


def test_one_column(orc):
    # Every product of a row meets in one column; 256 left steps.
    rng = np.random.default_rng(5)
    A = _rows(rng, 300, 1, 1, 1)
    R = _rows(rng, 16384, 300, 250, 256)
    _check(orc, [R, A], what="pair")


@pytest.mark.parametrize("M", [1, 31, 33, 127, 128, 129, 1000])
@pytest.mark.parametrize("k,l", [(8, 4), (31, 1), (1, 32), (3, 7)])
def test_tiny_rows(orc, M, k, l):
    rng = np.random.default_rng(100 * M + k)
    _check(orc, [_rows(rng, M, 50, 0, k), _rows(rng, 50, 40, min(l, 1), l)], what=(M, k, l))


def test_tiny_rows_all_distinct(orc):
    # 32 products, 32 columns: the list at its capacity.
    n = 32
    A = S.CSR(np.array([0, 8, 16]), np.tile(np.arange(8), 2), np.arange(16.0) - 7, (2, 8))
    B = S.CSR(np.arange(9) * 4, np.arange(n)[::1].astype(np.int64), np.arange(32.0) + 0.5, (8, n))
    _check(orc, [A, B])


@pytest.mark.parametrize("a_cols", [1, 600])
def test_booking_space_overflows(orc, a_cols):
    # More entries than the booking space holds (twice the operands', at
    # least 2^20): the product is redone with symbolic sizes, on the bounded
    # path (one product per row of R*A) and the binned one (600).
    rng = np.random.default_rng(6)
    R = _rows(rng, 2000, 1, 1, 1)
    A = _rows(rng, 1, a_cols, a_cols, a_cols)
    P = _rows(rng, a_cols, 600, 600 if a_cols == 1 else 1, 600 if a_cols == 1 else 1)
    if a_cols > 1:
        P = S.CSR(P.indptr, np.arange(600, dtype=np.int64), P.data, P.shape)
    _check(orc, [R, A, P])


@pytest.mark.parametrize("a_cols", [1, 600])
def test_galerkin_booking_space_overflows(orc, a_cols):
    # The same for operands that look like R = P^T (as many rows as P has
    # columns, as many entries), whose space is the operands' nonzeros once.
    rng = np.random.default_rng(9)
    R = _rows(rng, 1100, 1, 1, 1)
    A = _rows(rng, 1, a_cols, a_cols, a_cols)
    ptr = np.unique(np.linspace(0, 1100, a_cols + 1).astype(np.int64))
    P = S.CSR(ptr, np.arange(1100, dtype=np.int64), rng.uniform(-1.0, 1.0, 1100), (a_cols, 1100))
    _check(orc, [R, A, P])


@pytest.mark.parametrize("vt", [S.F64, S.F32])
@pytest.mark.parametrize("fl", [S.UB, S.SYMBNUM])
def test_batches(fl, vt):
    # Batches whose direct products are replayed (2D and 3D stencils, broken
    # patterns, fewer rows than a run) beside others (SpMM, heavy rows): equal
    # to the single products, also after new values.
    rng = np.random.default_rng(8)
    probs = [pb.stencil_problem(len(d), d) for d in
             [(170, 165), (41, 38, 35), (300, 120), (11, 9), (9, 8, 7), (64, 61), (47, 45, 40)]]
    ops = [[p.R, p.A, p.P] for p in probs]
    m = ops[2][1].to_scipy().copy()
    m.data[rng.random(m.nnz) < 0.01] = 0.0
    m.eliminate_zeros()
    ops[2][1] = S.CSR.from_scipy(m)
    ops.append([_rows(rng, 300, 400, 0, 40), _rows(rng, 400, 500, 0, 60), _rows(rng, 500, 90, 1, 9)])
    with S.Context() as ctx:
        for direct_only in (True, False):
            d = [[ctx.upload(_random_values(x, rng), vt) for x in o] for o in ops]
            if not direct_only:
                d.append([ctx.upload(_random_values(x, rng), vt) for x in ops[0][:2]])
            b = ctx.batch([tuple(x) for x in d], vt, fl)
            b.run()
            for step in range(2):
                for i, x in enumerate(d):
                    C = (ctx.rap(*x, S.DIRECT, S.UB, vt) if len(x) == 3 else
                         ctx.spmm(*x, S.UB, vt))
                    _equal(b.result(i).download(), C.download(), (direct_only, step, i))
                    C.free()
                for x in d:
                    x[1].set_values(rng.uniform(-1, 1, x[1].nnz).astype(
                        np.float64 if vt == S.F64 else np.float32).astype(np.float64))
                b.run()          # replays the numeric pass with the new values
            b.free()
            for x in d:
                for y in x:
                    y.free()
