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


def _cubes():
    import scipy.sparse as sp
    from sp3mm4amg_b200 import problems as pb
    rng = np.random.default_rng(3)

    def rand(M, N, lo, hi):
        n = rng.integers(lo, hi + 1, M)
        row = np.repeat(np.arange(M), n)
        m = sp.csr_matrix((rng.uniform(-1, 1, len(row)), (row, rng.integers(0, N, len(row)))),
                          shape=(M, N))
        m.sum_duplicates()
        m.sort_indices()
        return S.CSR(m.indptr.astype(np.int64), m.indices.astype(np.int64), m.data, m.shape)

    box, grid = pb.poisson3d(44), pb.poisson2d(320)
    A, P = rand(60000, 60000, 6, 8), rand(60000, 30000, 2, 4)
    return {"7-point cubed": [box] * 3, "5-point cubed": [grid] * 3,
            "random Galerkin": [P.transpose(), A, P],
            "random bounded": [rand(60000, 60000, 3, 6), rand(60000, 60000, 5, 15),
                               rand(60000, 30000, 1, 3)]}


@pytest.mark.parametrize("which", ["7-point cubed", "5-point cubed", "random Galerkin",
                                   "random bounded"])
def test_results_of_several_times_the_operands(orc, which):
    # Results of 1.6 to 7 times their operands' nonzeros (and more than 2^20),
    # also where R and P have the shapes and lengths of transposes.
    ops = _cubes()[which]
    want = orc.sp3mm_direct(*ops)
    assert want.nnz > 1.6 * sum(m.nnz for m in ops) and want.nnz > 1 << 20
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in ops]
        C, labels = _passes(ctx, lambda: ctx.rap(*d, S.DIRECT, S.UB))
        assert _booked_once(labels), labels
        _same(C, want, which)
        C.free()
        for m in d:
            m.free()


@pytest.mark.parametrize("kind", ["grid", "wide band"])
def test_hierarchies_book_enough(kind):
    # One level of a grid (less space booked) and of a band whose product holds
    # over twice its operands' nonzeros.
    from sp3mm4amg_b200 import problems as pb
    rng = np.random.default_rng(4)
    if kind == "grid":
        dims = (90, 80, 70)
        A = pb.poisson3d(*dims)
    else:
        import scipy.sparse as sp
        n = 100000
        dims = (n,)
        row = np.repeat(np.arange(n), 4)
        col = np.clip(row + rng.integers(-60, 61, 4 * n), 0, n - 1)
        m = sp.csr_matrix((rng.uniform(-1, 1, 4 * n), (row, col)), shape=(n, n))
        m = (m + m.T + 10 * sp.eye(n)).tocsr()
        m.sort_indices()
        A = S.CSR(m.indptr.astype(np.int64), m.indices.astype(np.int64), m.data, m.shape)
    with S.Context() as ctx:
        d = ctx.upload(A)
        ctx.set_profiling(True)
        h = ctx.hierarchy(d, dims, max_levels=2)
        labels = set(ctx.profile())
        ctx.set_profiling(False)
        assert _booked_once({x for x in labels if x.startswith("direct.")}), labels
        h.free()
        d.free()


def _pool_peak(ctx, f):
    """Most bytes in use in the device's memory pool during f(), above those
    in use before."""
    from cuda.bindings import driver, runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1] if len(r) > 1 else None

    attr = rt.cudaMemPoolAttr
    ctx.sync()
    pool = ok(rt.cudaDeviceGetDefaultMemPool(0))
    ok(rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, driver.cuuint64_t(0)))
    before = int(ok(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)))
    f()
    ctx.sync()
    return int(ok(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh))) - before


@pytest.mark.parametrize("variant", [S.DIRECT, S.PAIR])
def test_space_of_uneven_rows(variant):
    # One left row of 64 entries among 600,000 of one: the rows' bound (64
    # times 8 products) is 60 times what the operands allow.  The space stays
    # within the call's memory estimate.
    rng = np.random.default_rng(5)
    M, N = 600000, 500000
    n = np.ones(M, np.int64)
    n[M // 2] = 64
    ptr = np.concatenate([[0], np.cumsum(n)])
    R = S.CSR(ptr, np.concatenate([np.sort(rng.choice(N, 64, replace=False)) if k > 1 else
                                   rng.integers(0, N, 1) for k in n]).astype(np.int64),
              rng.uniform(-1, 1, int(ptr[-1])), (M, N))
    A = S.CSR(np.arange(N + 1, dtype=np.int64) * 8,
              (np.arange(N)[:, None] + np.arange(8)).ravel().astype(np.int64),
              rng.uniform(-1, 1, 8 * N), (N, N + 8))
    P = S.CSR(np.arange(N + 9, dtype=np.int64), np.arange(N + 8, dtype=np.int64),
              np.ones(N + 8), (N + 8, N + 8))
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in (R, A, P)]
        got = []
        peak = _pool_peak(ctx, lambda: got.append(ctx.rap(*d, variant, S.UB)))
        assert peak <= ctx.rap_memory_estimate(*d, variant, S.UB), peak
        # (its result holds 8 entries a row: 96 bytes, and as many booked)
        assert got[0].nnz > 7 * M
        got[0].free()
        for m in d:
            m.free()


def test_space_of_a_small_batch(orc):
    # A batch books no more than its results can hold: here 2 MB at most, not
    # the 12 MB of the least that larger batches take.
    from sp3mm4amg_b200 import problems as pb
    p = pb.stencil_problem(2, (50, 60))
    ops = (p.R, p.A, p.P)
    with S.Context() as ctx:
        d = [ctx.upload(m) for m in ops]
        got = []

        def run():
            got.append(ctx.batch([tuple(d), (d[0], d[1])]))
            got[0].run()
        peak = _pool_peak(ctx, run)
        assert peak < 6 << 20, peak
        for i, want in enumerate((orc.sp3mm_direct(*ops), orc.spmm(*ops[:2]))):
            cmp = O.compare(got[0].result(i).download(), want, rtol=0.0)
            assert cmp["ok"] and cmp["bitwise_equal"] == want.nnz, (i, cmp)
        got[0].free()
        for m in d:
            m.free()
