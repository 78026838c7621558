"""The work an AMG setup does with this package, as cases to be measured.

A user forms coarse operators C = R*A*P: one product at a time with operands
that stay on the device (either variant and flavour, FP64 or FP32 storage,
regular grids and irregular graphs), many small products in one batch, whole
hierarchies one at a time or many together, and single products from host
matrices through the reference-named C entry points.

Operators are variable-coefficient diffusion operators on box grids (5-point
in 2D, 7-point in 3D, a seeded conductivity per cell face, Dirichlet
boundary) and k-nearest-neighbour graph Laplacians; prolongators are block
(or greedy) aggregation smoothed by one damped-Jacobi step.  Another seed
gives another operator of the same size.
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

import sp3mm4amg_b200 as S
from sp3mm4amg_b200 import capi, problems
from sp3mm4amg_b200.spmat import CONFIG, RBTREE, HostSpMat, csr_from_spmat, SPMAT_P

OMEGA = 2.0 / 3.0
MIN_COARSE = 1000        # a hierarchy's coarsest level has fewer rows than this
VARIANTS = {"direct": S.DIRECT, "pair": S.PAIR, "pair_right": S.PAIR_RIGHT}
FLAVOURS = {"ub": S.UB, "symbnum": S.SYMBNUM}
VALUES = {"f64": S.F64, "f32": S.F32}


def listed():
    return [
        # The smallest setup call: a 64x64 grid's finest product, where
        # launches and round trips count.
        {"name": "direct_2d_64", "kind": "rap", "nx": 64, "ny": 64, "nz": 0,
         "variant": "direct", "flavour": "ub", "values": "f64"},
        # An ordinary 2D product on a ragged grid (partial blocks at both
        # edges), with exact symbolic sizes instead of booked upper bounds.
        {"name": "direct_2d_ragged", "kind": "rap", "nx": 517, "ny": 389, "nz": 0,
         "variant": "direct", "flavour": "symbnum", "values": "f64"},
        # The headline product: the finest level of a 128^3 problem.
        {"name": "direct_3d_128", "kind": "rap", "nx": 128, "ny": 128, "nz": 128,
         "variant": "direct", "flavour": "ub", "values": "f64"},
        # The pair-wise products (R*A)*P, the reference's fastest variant, on
        # an ordinary odd 3D box with symbolic sizes.
        {"name": "pair_3d_odd", "kind": "rap", "nx": 61, "ny": 47, "nz": 53,
         "variant": "pair", "flavour": "symbnum", "values": "f64"},
        # R*(A*P) with FP32 storage, as coarse levels may be kept.
        {"name": "pair_right_3d_f32", "kind": "rap", "nx": 96, "ny": 80, "nz": 88,
         "variant": "pair_right", "flavour": "ub", "values": "f32"},
        # An irregular operator: uneven rows, no grid order, greedy aggregates.
        {"name": "direct_knn", "kind": "knn", "points": 80000, "k": 16,
         "variant": "direct", "flavour": "ub", "values": "f64"},
        # A whole 128^3 hierarchy: prolongators, restrictions and Galerkin
        # products of every level, the coarse ones with rows of hundreds of
        # entries.
        {"name": "hierarchy_3d_128", "kind": "hierarchy", "nx": 128, "ny": 128, "nz": 128,
         "coarse": "f64"},
        # A 2D hierarchy on a ragged grid with FP32 coarse storage.
        {"name": "hierarchy_2d_f32", "kind": "hierarchy", "nx": 447, "ny": 433, "nz": 0,
         "coarse": "f32"},
        # Many small and middling hierarchies built level by level together,
        # as the setup server does with the requests it holds.
        {"name": "hierarchies_24", "kind": "hierarchies", "count": 24, "specs": 3,
         "nmin": 1000, "nmax": 200000, "coarse": "f64"},
        # One batch of uneven products, as a program with new patterns runs
        # it: the batch is made, planned and executed.
        {"name": "batch_run_20", "kind": "batch_run", "count": 20, "specs": 7,
         "nmin": 1000, "nmax": 200000},
        # The numeric re-setup of a planned batch: patterns kept, values read anew.
        {"name": "batch_replay_20", "kind": "batch_replay", "count": 20, "specs": 11,
         "nmin": 1000, "nmax": 200000},
        # A reference user's call: host matrices in malloc'd memory through
        # the reference-named entry point, the result back on the host.
        {"name": "host_direct", "kind": "host", "nx": 72, "ny": 60, "nz": 68,
         "entry": "sp3mmRowByRowMerged_0"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, nmin, nmax):
    """An uneven 2D or 3D box of nmin to nmax points."""
    n = _log(rng, nmin, nmax)
    if rng.random() < 0.4:
        nx = max(8, int(round(math.sqrt(n) * rng.uniform(0.75, 1.3))))
        return {"nx": nx, "ny": max(8, n // nx), "nz": 0}
    nx = max(5, int(round(n ** (1 / 3) * rng.uniform(0.8, 1.25))))
    ny = max(5, int(round(n ** (1 / 3) * rng.uniform(0.8, 1.25))))
    return {"nx": nx, "ny": ny, "nz": max(5, n // (nx * ny))}


def draw(rng):
    kind = rng.choice(["rap", "rap", "rap", "rap", "knn", "hierarchy", "hierarchies",
                       "batch_run", "batch_replay", "host"])
    if kind == "rap":
        return {"kind": kind, **_grid(rng, 4096, 2000000),
                "variant": rng.choice(["direct", "direct", "pair", "pair_right"]),
                "flavour": rng.choice(["ub", "symbnum"]),
                "values": rng.choice(["f64", "f64", "f32"])}
    if kind == "knn":
        return {"kind": kind, "points": _log(rng, 8000, 90000), "k": rng.choice([8, 12, 16]),
                "variant": rng.choice(["direct", "pair"]),
                "flavour": rng.choice(["ub", "symbnum"]), "values": "f64"}
    if kind == "hierarchy":
        return {"kind": kind, **_grid(rng, 8000, 1500000), "coarse": rng.choice(["f64", "f32"])}
    if kind == "host":
        return {"kind": kind, **_grid(rng, 4096, 300000),
                "entry": rng.choice(["sp3mmRowByRowMerged_0", "sp3mmRowByRowPair_0"])}
    case = {"kind": kind, "count": rng.randint(6, 20), "specs": rng.randint(100, 10 ** 6),
            "nmin": 1000, "nmax": 200000}
    if kind == "hierarchies":
        case["coarse"] = rng.choice(["f64", "f32"])
    return case


# ---------------------------------------------------------------------------
# Inputs.

def _dims(case):
    return tuple(case[a] for a in ("nx", "ny", "nz") if case[a])


def _batch_dims(case):
    rng = random.Random(case["specs"])
    return [tuple(v for v in _grid(rng, case["nmin"], case["nmax"]).values() if v)
            for _ in range(case["count"])]


def _diffusion(dims, seed):
    """Variable-coefficient diffusion on a box grid: x fastest, -conductivity
    off the diagonal, the sum of the cell's faces on it."""
    rng = np.random.default_rng(seed)
    d = len(dims)
    shape = tuple(reversed(dims))           # slowest axis first
    n = int(np.prod(dims))
    stride = [int(np.prod(shape[a + 1:])) for a in range(d)]
    lo, hi, has_lo, has_hi = [], [], [], []
    for a in range(d):
        fs = list(shape)
        fs[a] += 1
        face = rng.uniform(0.5, 1.5, fs)
        lo.append(np.take(face, range(shape[a]), axis=a))
        hi.append(np.take(face, range(1, shape[a] + 1), axis=a))
        at = np.arange(shape[a]).reshape([-1 if b == a else 1 for b in range(d)])
        has_lo.append(np.broadcast_to(at > 0, shape))
        has_hi.append(np.broadcast_to(at < shape[a] - 1, shape))
    val = np.empty((n, 2 * d + 1))
    keep = np.empty((n, 2 * d + 1), bool)
    for a in range(d):
        val[:, a], keep[:, a] = -lo[a].ravel(), has_lo[a].ravel()
        val[:, 2 * d - a], keep[:, 2 * d - a] = -hi[a].ravel(), has_hi[a].ravel()
    val[:, d], keep[:, d] = sum(lo).ravel() + sum(hi).ravel(), True
    off = np.array([-s for s in stride] + [0] + stride[::-1], np.int64)
    col = np.arange(n, dtype=np.int64)[:, None] + off
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(keep.sum(1), out=ptr[1:])
    return S.CSR(ptr, col[keep], val[keep], (n, n))


@functools.lru_cache(maxsize=8)
def _graph(points, k):
    """A k-nearest-neighbour graph (a CSR with a diagonal), the number of
    each entry's undirected edge (0 on the diagonal) and its aggregation."""
    A, _ = problems.knn_laplacian(points, k, seed=2)
    P0 = problems.aggregates_from_labels(problems.greedy_aggregation(A, seed=2))
    row = np.repeat(np.arange(A.M, dtype=np.int64), np.diff(A.indptr))
    off = row != A.indices
    lo, hi = np.minimum(row, A.indices)[off], np.maximum(row, A.indices)[off]
    edge = np.zeros(A.nnz, np.int64)
    edge[off] = np.unique(lo * A.M + hi, return_inverse=True)[1]
    return A, row, off, edge, P0


def _knn(case, seed):
    """Restriction, graph Laplacian and prolongator: the graph and its
    aggregation belong to the case, the edge weights to the seed."""
    G, row, off, edge, P0 = _graph(case["points"], case["k"])
    weight = np.random.default_rng(seed).uniform(0.5, 1.5, int(edge.max()) + 1)
    val = np.where(off, -weight[edge], 0.0)
    val[~off] = np.bincount(row, weights=-val, minlength=G.M) + 1e-3
    A = S.CSR(G.indptr, G.indices, val, G.shape)
    P = problems.jacobi_smooth(A, P0, OMEGA)
    return P.transpose(), A, P


_CTX = []


def _context():
    """The program's device context, on a torch stream so that torch
    operations on results can be ordered after the products."""
    if not _CTX:
        stream = torch.cuda.Stream()
        _CTX.extend((S.Context(stream=stream.cuda_stream), stream))
    return _CTX


class _Owned:
    """A device object of the package, freed with its last reference."""

    def __init__(self, *objects):
        self.objects = objects

    def free(self):
        for o in self.objects:
            o.free()
        self.objects = ()

    def __del__(self):
        self.free()


class _Memory:
    def __init__(self, ptr, n, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr,
                                         "data": (ptr if n else 0, False), "version": 3}


def _arrays(m, owner):
    """Tensors over a DeviceCSR's arrays; they keep `owner` alive."""
    def tensor(ptr, n, typestr):
        return torch.as_tensor(_Memory(ptr, n, typestr, owner), device="cuda")
    return {"row_ptr": tensor(m.d.row_ptr, m.shape[0] + 1, "<i4"),
            "col": tensor(m.d.col, m.nnz, "<i4"),
            "val": tensor(m.d.val, m.nnz, "<f4" if m.val_type == S.F32 else "<f8")}


class _State:
    def __init__(self, case, **have):
        self.case = case
        self.__dict__.update(have)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host":
        dims = _dims(case)
        A = _diffusion(dims, seed)
        P = problems.jacobi_smooth(A, problems.block_aggregation(dims), OMEGA)
        mats = [HostSpMat(m) for m in (P.transpose(), A, P)]
        return _State(case, mats=mats, lib=capi.load(), libc=ctypes.CDLL(None),
                      cfg=CONFIG(gridRows=20, gridCols=2, symbMMRowImplID=RBTREE, threadNum=1,
                                 chunkDistrbFunc=None))
    ctx, stream = _context()
    if kind == "knn":
        ops = [ctx.upload(m) for m in _knn(case, seed)]
        return _State(case, ctx=ctx, ops=ops, owner=_Owned(*ops))
    if kind == "rap":
        vt = VALUES[case["values"]]
        ops = _galerkin(ctx, _dims(case), seed, vt)
        return _State(case, ctx=ctx, ops=ops, owner=_Owned(*ops))
    if kind == "hierarchy":
        A = ctx.upload(_diffusion(_dims(case), seed))
        return _State(case, ctx=ctx, A=A, owner=_Owned(A))
    dims = _batch_dims(case)
    if kind == "hierarchies":
        As = [ctx.upload(_diffusion(d, 1000 * seed + i)) for i, d in enumerate(dims)]
        return _State(case, ctx=ctx, stream=stream, As=As, dims=dims, owner=_Owned(*As))
    products = [tuple(_galerkin(ctx, d, 1000 * seed + i, S.F64)) for i, d in enumerate(dims)]
    owner = _Owned(*[m for p in products for m in p])
    if kind == "batch_run":
        return _State(case, ctx=ctx, products=products, owner=owner)
    batch = ctx.batch(products)
    batch.plan()
    owner = _Owned(batch, owner)
    return _State(case, ctx=ctx, batch=batch, owner=owner,
                  out=[_arrays(batch.result(i), owner) for i in range(len(batch))])


def _galerkin(ctx, dims, seed, vt):
    A = ctx.upload(_diffusion(dims, seed), vt)
    P = ctx.block_prolongator(A, dims, out_val_type=vt)
    return [ctx.transpose(P), A, P]


# ---------------------------------------------------------------------------
# One pass.

def run(state):
    case = state.case
    kind = case["kind"]
    if kind in ("rap", "knn"):
        C = state.ctx.rap(*state.ops, variant=VARIANTS[case["variant"]],
                          flavour=FLAVOURS[case["flavour"]], out_val_type=VALUES[case["values"]])
        return _arrays(C, _Owned(C))
    if kind == "hierarchy":
        h = state.ctx.hierarchy(state.A, _dims(case), omega=OMEGA, min_coarse=MIN_COARSE,
                                max_levels=20, coarse_val_type=VALUES[case["coarse"]])
        return _levels(h, _Owned(h))
    if kind == "hierarchies":
        hs = state.ctx.hierarchies(state.As, state.dims, omega=OMEGA, min_coarse=MIN_COARSE,
                                   max_levels=20, coarse_val_type=VALUES[case["coarse"]])
        owner = _Owned(*hs)
        return _packed([_levels(h, owner) for h in hs], state.stream)
    if kind == "batch_run":
        batch = state.ctx.batch(state.products)
        owner = _Owned(batch)
        batch.run()
        return [_arrays(batch.result(i), owner) for i in range(len(batch))]
    if kind == "batch_replay":
        state.batch.execute()
        return state.out
    f = getattr(state.lib, case["entry"])
    p = f(*[m.ptr for m in state.mats], ctypes.byref(state.cfg), None)
    if not p:
        raise RuntimeError(case["entry"] + " returned NULL")
    C = csr_from_spmat(p, 0)
    m = ctypes.cast(p, SPMAT_P).contents
    for a in (m.AS, m.JA, m.IRP):
        state.libc.free(ctypes.cast(a, ctypes.c_void_p))
    state.libc.free(ctypes.c_void_p(p))
    return {"row_ptr": C.indptr, "col": C.indices, "val": C.data}


def _levels(h, owner):
    """Every matrix a hierarchy build makes: A of each coarse level, P and R."""
    out = []
    for level in range(len(h)):
        A, P, R = h.level(level)
        for name, m in (("A", A if level else None), ("P", P), ("R", R)):
            if m is not None:
                out.append({"name": name + str(level), **_arrays(m, owner)})
    return {m.pop("name"): m for m in out}


def _packed(hierarchies, stream):
    """All hierarchies' matrices one after another, the values by the type
    they are stored in."""
    mats = [m for h in hierarchies for m in h.values()]
    with torch.cuda.stream(stream):
        out = {k: torch.cat([m[k] for m in mats]) for k in ("row_ptr", "col")}
        for dtype in {m["val"].dtype for m in mats}:
            out[str(dtype)] = torch.cat([m["val"] for m in mats if m["val"].dtype == dtype])
    return out


# ---------------------------------------------------------------------------
# The same in 64 bits with torch alone, and the work it is.

class _Csr:
    """A sparse matrix as torch tensors (64-bit indices, FP64 values)."""

    def __init__(self, ptr, col, val, cols):
        self.ptr, self.col, self.val, self.cols = ptr, col, val, cols

    @property
    def rows(self):
        return self.ptr.numel() - 1

    @property
    def nnz(self):
        return self.col.numel()

    def row_of(self):
        return torch.repeat_interleave(torch.arange(self.rows, device=self.ptr.device),
                                       self.ptr.diff())

    def out(self):
        return {"row_ptr": None, "col": None, "val": self.val}

    def bytes(self, value=8):
        return (self.rows + 1) * 4 + self.nnz * (4 + value)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _torch_csr(m, f32=False):
    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(_device())
    v = t(m.data)
    return _Csr(t(m.indptr), t(m.indices), v.float().double() if f32 else v, m.N)


def _from_keys(rows, cols, key, val):
    """CSR of summed entries; `key` = row * cols + column."""
    uniq, where = torch.unique(key, return_inverse=True)
    out = torch.zeros(uniq.numel(), dtype=torch.float64, device=key.device)
    out.index_add_(0, where, val)
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device=key.device)
    ptr[1:] = torch.bincount(uniq // cols, minlength=rows).cumsum(0)
    return _Csr(ptr, uniq % cols, out, cols)


def _product(A, B, most=1 << 26):
    """(A*B, multiply-adds), expanded and summed `most` products at a time."""
    lens = B.ptr.diff()[A.col]
    ends = lens.cumsum(0)
    total = int(ends[-1]) if ends.numel() else 0
    before = torch.cat([ends.new_zeros(1), ends])[A.ptr]    # products before each row
    parts, first = [], 0
    while first < A.rows:
        last = int(torch.searchsorted(before, before[first] + most, right=True)) - 1
        last = min(max(last, first + 1), A.rows)
        s, e = int(A.ptr[first]), int(A.ptr[last])
        ln = lens[s:e]
        entry = torch.repeat_interleave(torch.arange(e - s, device=ln.device), ln)
        at = torch.arange(entry.numel(), device=ln.device) - (ln.cumsum(0) - ln)[entry]
        at += B.ptr[A.col[s:e]][entry]
        row = torch.repeat_interleave(torch.arange(last - first, device=ln.device),
                                      A.ptr[first:last + 1].diff())
        parts.append(_from_keys(last - first, B.cols, row[entry] * B.cols + B.col[at],
                                A.val[s:e][entry] * B.val[at]))
        first = last
    ptr = torch.cat([A.ptr.new_zeros(1), torch.cat([p.ptr.diff() for p in parts]).cumsum(0)])
    return _Csr(ptr, torch.cat([p.col for p in parts]), torch.cat([p.val for p in parts]),
                B.cols), total


def _transpose(A):
    col, order = torch.sort(A.col, stable=True)
    ptr = torch.zeros(A.cols + 1, dtype=torch.int64, device=col.device)
    ptr[1:] = torch.bincount(col, minlength=A.cols).cumsum(0)
    return _Csr(ptr, A.row_of()[order], A.val[order], A.rows)


def _prolongator(A, dims):
    """(I - omega D^-1 A) P0 for 2^d block aggregation; the coarse box."""
    cdims = tuple(-(-d // 2) for d in dims)
    rem = torch.arange(A.rows, device=A.ptr.device)
    agg, stride = torch.zeros_like(rem), 1
    for d, cd in zip(dims, cdims):
        agg += (rem % d) // 2 * stride
        rem = rem // d
        stride *= cd
    row = A.row_of()
    diag = torch.zeros(A.rows, dtype=torch.float64, device=row.device)
    on = A.col == row
    diag[row[on]] = A.val[on]
    P = _from_keys(A.rows, stride, row * stride + agg[A.col], A.val)
    row = P.row_of()
    P.val = (P.col == agg[row]).double() - (OMEGA / diag)[row] * P.val
    return P, cdims


def _triple(case, seed):
    f32 = case.get("values") == "f32"
    if case["kind"] == "knn":
        return [_torch_csr(m) for m in _knn(case, seed)]
    A = _torch_csr(_diffusion(_dims(case), seed), f32)
    P, _ = _prolongator(A, _dims(case))
    if f32:
        P.val = P.val.float().double()
    return [_transpose(P), A, P]


def _chain(A, dims):
    """The matrices of a hierarchy by name, and its products' multiply-adds."""
    out, flops, level = {}, 0, 0
    while A.rows >= MIN_COARSE and A.rows > 1 and level < 19:
        P, dims = _prolongator(A, dims)
        R = _transpose(P)
        T, n1 = _product(R, A)
        C, n2 = _product(T, P)
        flops += 2 * (n1 + n2)
        if level:
            out["A%d" % level] = A
        out["P%d" % level], out["R%d" % level] = P, R
        A, level = C, level + 1
    if level:
        out["A%d" % level] = A
    return out, flops


def _pieces(case, seed):
    """(dims, operator seed) of each problem of a case on several grids."""
    return [(d, 1000 * seed + i) for i, d in enumerate(_batch_dims(case))]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rap", "knn", "host"):
        R, A, P = _triple(case, seed)
        return _product(_product(R, A)[0], P)[0].out()
    if kind == "hierarchy":
        mats, _ = _chain(_torch_csr(_diffusion(_dims(case), seed)), _dims(case))
        return {name: m.out() for name, m in mats.items()}
    if kind == "hierarchies":
        vals = {"torch.float64": [], "torch.float32": []}
        for dims, s in _pieces(case, seed):
            for name, m in _chain(_torch_csr(_diffusion(dims, s)), dims)[0].items():
                # Level 0's prolongator and restriction are FP64 in both modes.
                fine = case["coarse"] == "f64" or name in ("P0", "R0")
                vals["torch.float64" if fine else "torch.float32"].append(m.val)
        return {"row_ptr": None, "col": None,
                **{k: torch.cat(v) for k, v in vals.items() if v}}
    out = []
    for dims, s in _pieces(case, seed):
        A = _torch_csr(_diffusion(dims, s))
        P, _ = _prolongator(A, dims)
        out.append(_product(_product(_transpose(P), A)[0], P)[0].out())
    return out


def work(case):
    kind = case["kind"]
    if kind in ("rap", "knn", "host"):
        v = 4 if case.get("values") == "f32" else 8
        R, A, P = _triple(case, 0)
        T, n1 = _product(R, A)
        C, n2 = _product(T, P)
        if kind == "host":   # 64-bit indices, as the caller holds them
            return {"bytes": sum((m.rows + 1) * 8 + m.nnz * 16 for m in (R, A, P, C)),
                    "flops": 2 * (n1 + n2)}
        return {"bytes": sum(m.bytes(v) for m in (R, A, P, C)), "flops": 2 * (n1 + n2)}
    grids = [(_dims(case), 0)] if kind == "hierarchy" else _pieces(case, 0)
    nbytes = flops = 0
    for dims, s in grids:
        A = _torch_csr(_diffusion(dims, s))
        if kind in ("hierarchy", "hierarchies"):
            v = 4 if case["coarse"] == "f32" else 8
            mats, n = _chain(A, dims)
            nbytes += A.bytes() + sum(m.bytes(8 if name in ("P0", "R0") else v)
                                      for name, m in mats.items())
            flops += n
        else:
            P, _ = _prolongator(A, dims)
            R = _transpose(P)
            T, n1 = _product(R, A)
            C, n2 = _product(T, P)
            nbytes += sum(m.bytes() for m in (R, A, P, C))
            flops += 2 * (n1 + n2)
    return {"bytes": nbytes, "flops": flops}
