"""Rows whose paged stage-1 slice runs out of pages (rowdense.cuh): the steps
end early and the row walks its span in chunks, with the same result, at little
more than the chunks' own time."""
import numpy as np
import pytest

import sp3mm4amg_b200 as S
from test_gpu_dense import DENSE, _direct_all_ways

pytestmark = pytest.mark.gpu


def _scattered(rng, N, columns, run, M, steps=200, entries=100):
    """R*A rows of `steps` A rows, each `entries` columns in runs of `run` out of
    about `columns` spread over N."""
    start = np.sort(rng.choice((N - run) // run, columns // run, replace=False)) * run
    rows = [np.unique((rng.choice(start, entries // run, replace=False)[:, None] +
                       np.arange(run)).ravel()) for _ in range(1000)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    A = S.CSR(ptr, np.concatenate(rows).astype(np.int64), rng.uniform(-1, 1, int(ptr[-1])),
              (1000, N))
    cols = np.sort(np.argsort(rng.random((M, 1000)), axis=1)[:, :steps], axis=1)
    R = S.CSR(np.arange(M + 1, dtype=np.int64) * steps, cols.ravel().astype(np.int64),
              rng.uniform(-1, 1, M * steps), (M, 1000))
    P = S.CSR(np.arange(N + 1, dtype=np.int64), np.arange(N, dtype=np.int64) % 500,
              rng.uniform(-1, 1, N), (N, 500))
    return R, A, P


@pytest.mark.parametrize("N,columns,run,steps,entries", [
    (12000, 1800, 1, 200, 100),   # over half the pages' columns alone: late
    (30000, 1800, 3, 201, 100),   # some pages too few; not a multiple of four steps
    (60000, 3600, 1, 3, 1200),    # within the first steps; rows of several per thread
    (60000, 3000, 2, 600, 60),    # more steps than are described at a time
])
def test_pages_run_out(orc, N, columns, run, steps, entries):
    rng = np.random.default_rng(N + run)
    R, A, P = _scattered(rng, N, columns, run, 12, steps, entries)
    with S.Context() as ctx:
        _direct_all_ways(ctx, orc, R, A, P, (N, columns, run))
        _direct_all_ways(ctx, orc, R, A, P, (N, columns, run, "f32"), vt=S.F32)


def test_time_of_scattered_columns():
    # The same products over a span within one slice and over one of two: one
    # pass against two (1.3 times as long by the whole kernel; 1.9 with a third
    # pass spent on the pages).
    t = {}
    with S.Context() as ctx:
        for N in (8000, 12000):
            d = [ctx.upload(m) for m in _scattered(np.random.default_rng(1), N, 1800, 1, 900)]
            ctx.set_tuning(DENSE)
            for _ in range(4):
                ctx.set_profiling(True)
                ctx.rap(*d, S.DIRECT, S.UB).free()
                ms = ctx.profile()["direct.dense.book"][1]
                ctx.set_profiling(False)
                t[N] = min(t.get(N, ms), ms)
            ctx.set_tuning(0)
            for m in d:
                m.free()
    assert t[12000] < 1.7 * t[8000], t
