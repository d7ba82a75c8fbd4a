"""The work that users of this framework have it do, as cases that can be timed.

A case is one use of the public entry points on inputs that a program already
holds.  Matrices and vectors of the GraphBLAS API are resident in HBM before a
pass and their results stay there after it, as in a program that goes on to
use them; only the `round_trip` kind crosses the host boundary in the pass
itself.  Every call has finished when it returns (the API is synchronous).

Graphs are R-MAT with (a,b,c,d) = (0.57,0.19,0.19,0.05), symmetrised, without
self-loops and duplicates; a vertex count that is no power of two keeps the
edges among the first n vertices of the next larger graph.  "er" matrices have
a uniform number of entries in [dmin, dmax] per row at uniform columns.
"""

import functools
import math

import numpy as np
import torch

from graphblas_b200 import batch as B
from graphblas_b200 import semiring
from graphblas_b200 import workloads as W
from graphblas_b200.grb import API

# R-MAT quadrant probabilities of every graph here (graph500)
RMAT = (0.57, 0.19, 0.19, 0.05)
BOOL, INT64, FP32, FP64 = 1, 8, 10, 11
NP = {INT64: np.int64, FP32: np.float32, FP64: np.float64}
PRODUCT = {"plus_times_fp64": ("GrB_PLUS_TIMES_SEMIRING_FP64", FP64),
           "plus_times_fp32": ("GrB_PLUS_TIMES_SEMIRING_FP32", FP32),
           "min_plus_fp32": ("GrB_MIN_PLUS_SEMIRING_FP32", FP32)}


def listed():
    return [
        # Triangle counting (LAGraph's Sandia-LUT: C<L> = L*U' plus_pair, then
        # the sum).  A small community graph, where the call's launches count,
        {"name": "triangles_1k", "kind": "triangles", "n": 1024, "ef": 16},
        # and the graph500 scale-20 graph that triangle rates are quoted on.
        {"name": "triangles_1m", "kind": "triangles", "n": 1 << 20, "ef": 16},
        # Edge similarity: C<A> = A*A' in plus_times fp64 over A's own pattern
        # (cosine / common-neighbour weights): masked dot products that are
        # no plain counts.
        {"name": "similarity_16k", "kind": "similarity", "n": 16384, "ef": 16},
        # Sparse products A*A on evenly filled matrices: the smallest that a
        # request server sees,
        {"name": "product_er_1k", "kind": "product", "graph": "er", "n": 1000, "dmin": 4,
         "dmax": 16, "semiring": "plus_times_fp64"},
        # the ordinary one (8 entries in every row),
        {"name": "product_er_16k", "kind": "product", "graph": "er", "n": 16384, "dmin": 8,
         "dmax": 8, "semiring": "plus_times_fp64"},
        # and the largest.
        {"name": "product_er_65k", "kind": "product", "graph": "er", "n": 65536, "dmin": 4,
         "dmax": 16, "semiring": "plus_times_fp64"},
        # A two-hop product of a skewed graph: rows from empty to hubs with
        # hundreds of thousands of products.
        {"name": "product_rmat_5k", "kind": "product", "graph": "rmat", "n": 5000, "ef": 16,
         "semiring": "plus_times_fp64"},
        # A product whose operands arrive in page-locked host memory and whose
        # result goes back there (GrB_Matrix_import, GrB_mxm,
        # GrB_Matrix_export).
        {"name": "round_trip_3k", "kind": "round_trip", "n": 3001, "dmin": 4, "dmax": 16},
        # Breadth-first search for parents: push only on a graph of ordinary
        # size, where every level's launches count,
        {"name": "bfs_push_50k", "kind": "bfs", "n": 50000, "ef": 16, "pull": False},
        # and direction-optimising on a large one.
        {"name": "bfs_pull_2m", "kind": "bfs", "n": 1 << 21, "ef": 16, "pull": True},
        # Hop-limited shortest paths: d = min(d, d min.+ A) in fp32.
        {"name": "sssp_260k", "kind": "sssp", "n": 260000, "ef": 16, "hops": 6},
        # Independent products in one batch (A_k*A_k, min_plus fp32).
        {"name": "batch_1000", "kind": "batch", "count": 1000, "nmax": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["triangles", "similarity", "product", "product", "round_trip", "bfs",
                       "bfs", "sssp", "batch"])
    if kind == "triangles":
        return {"kind": kind, "n": _log_int(rng, 600, 1 << 20), "ef": 16}
    if kind == "similarity":
        return {"kind": kind, "n": _log_int(rng, 600, 16384), "ef": rng.randint(8, 16)}
    if kind == "product":
        name = rng.choice(sorted(PRODUCT))
        if rng.random() < 0.7:
            dmin = rng.randint(2, 8)
            return {"kind": kind, "graph": "er", "n": _log_int(rng, 300, 65536), "dmin": dmin,
                    "dmax": rng.randint(dmin, 16), "semiring": name}
        return {"kind": kind, "graph": "rmat", "n": _log_int(rng, 500, 5000),
                "ef": rng.randint(8, 16), "semiring": name}
    if kind == "round_trip":
        return {"kind": kind, "n": _log_int(rng, 300, 20000), "dmin": 4, "dmax": 16}
    if kind == "bfs":
        return {"kind": kind, "n": _log_int(rng, 2000, 1 << 21), "ef": 16,
                "pull": rng.random() < 0.5}
    if kind == "sssp":
        return {"kind": kind, "n": _log_int(rng, 2000, 260000), "ef": 16,
                "hops": rng.randint(3, 6)}
    return {"kind": kind, "count": _log_int(rng, 40, 1000), "nmax": _log_int(rng, 500, 8192)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _csr_of_keys(keys, nrows, ncols):
    """(p, i) of the sorted keys row * ncols + column."""
    row = torch.div(keys, ncols, rounding_mode="floor")
    p = torch.zeros(nrows + 1, dtype=torch.int64, device=keys.device)
    p[1:] = torch.cumsum(torch.bincount(row, minlength=nrows), 0)
    return p, keys - row * ncols


def _rmat(n, ef, gen):
    """(p, i) of a symmetric R-MAT pattern on n vertices."""
    dev = _device()
    scale = max(1, (n - 1).bit_length())
    m = ef << scale
    a, b, c, _ = RMAT
    u = torch.zeros(m, dtype=torch.int64, device=dev)
    v = torch.zeros(m, dtype=torch.int64, device=dev)
    for _ in range(scale):
        r = torch.rand(m, device=dev, generator=gen)
        u = 2 * u + (r >= a + b)
        v = 2 * v + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    ok = (u != v) & (u < n) & (v < n)
    u, v = u[ok], v[ok]
    keys = torch.unique(torch.cat([u * n + v, v * n + u]))
    return _csr_of_keys(keys, n, n)


def _er(n, dmin, dmax, gen):
    """(p, i) of an n-by-n pattern, dmin to dmax distinct columns in a row."""
    dev = _device()
    deg = torch.randint(dmin, dmax + 1, (n,), device=dev, generator=gen)
    # a few columns more than asked for, so that enough distinct ones are left
    col = torch.randint(0, n, (n, 2 * dmax + 8), device=dev, generator=gen)
    srt, order = torch.sort(col, dim=1, stable=True)
    first = torch.ones_like(col, dtype=torch.bool)
    first[:, 1:] = srt[:, 1:] != srt[:, :-1]
    keep = torch.zeros_like(first).scatter_(1, order, first)     # first draws, in drawn order
    keep &= torch.cumsum(keep, 1) <= deg[:, None]
    row = torch.arange(n, device=dev)[:, None].expand_as(col)
    return _csr_of_keys(torch.sort((row * n + col)[keep])[0], n, n)


def _pattern(case, gen):
    if case.get("graph", "rmat") == "er" or case["kind"] == "round_trip":
        return _er(case["n"], case["dmin"], case["dmax"], gen)
    return _rmat(case["n"], case["ef"], gen)


def _values(nnz, code, gen, lo, hi):
    x = torch.rand(nnz, device=_device(), generator=gen, dtype=torch.float64) * (hi - lo) + lo
    return x.float() if code == FP32 else x


def _matrix(case, seed):
    """(p, i, x, type code) of the case's operand, torch tensors."""
    gen = _generator(seed)
    p, i = _pattern(case, gen)
    if case["kind"] == "sssp" or case.get("semiring") == "min_plus_fp32":
        return p, i, _values(len(i), FP32, gen, 0.1, 10.0), FP32
    code = PRODUCT[case.get("semiring", "plus_times_fp64")][1]
    return p, i, _values(len(i), code, gen, -1.0, 1.0), code


def _source(p, seed):
    """A vertex with an edge."""
    some = torch.nonzero(p[1:] > p[:-1]).flatten()
    return int(some[np.random.default_rng(seed).integers(len(some))])


@functools.lru_cache(maxsize=None)
def _api():
    return API()


def _import(p, i, x, code, n):
    """GrB_Matrix_import: the matrix is resident in HBM when it returns."""
    p, i, x = (np.ascontiguousarray(t.cpu().numpy()) for t in (p, i, x))
    return _api().matrix_import(code, n, n, p.ctypes.data, i.ctypes.data, x.ctypes.data, len(i))


@functools.lru_cache(maxsize=64)
def _sizes(count, nmax):
    return tuple(W.batch_sizes(count, 64, nmax))


def _batch_sizes(case):
    """Log-uniform sizes in [64, nmax]."""
    return _sizes(case["count"], case["nmax"])


def _batch(case, seed):
    """Poisson(6) entries a row, fp32 weights in [0.1, 10]."""
    return [W.poisson_minw(n, 6.0, 0.1, 10.0, (int(seed) * 100003 + k) % (1 << 62))
            for k, n in enumerate(_batch_sizes(case))]


def _ones(i):
    return torch.ones(len(i), dtype=torch.bool, device=i.device)


# ---------------------------------------------------------------------------
# results that stay on the device
# ---------------------------------------------------------------------------

class Resident(dict):
    """The arrays of a result that stays in HBM, copied out when asked for.
    Arrays of entries have a length that the case alone decides, the entries
    first and zeros after them; vectors come dense."""

    def __init__(self, names, read):
        super().__init__((k, None) for k in names)
        self._read = read

    def __getitem__(self, k):
        if self._read is not None:
            read, self._read = self._read, None
            self.update(read())
        return super().__getitem__(k)


def _room(case):
    """Entries that no result of the case goes past."""
    kind = case["kind"]
    if kind == "batch":
        return 64 * (sum(_batch_sizes(case)) + 64)        # 36 products a row are expected
    n = case["n"]
    if kind == "triangles":
        return case["ef"] << (n - 1).bit_length()
    if kind == "similarity":
        return 2 * case["ef"] << (n - 1).bit_length()
    if case.get("graph") == "rmat":
        return n * n
    return min(n * n, n * case["dmax"] ** 2)


def _padded(a, room):
    out = np.zeros(room, a.dtype)
    out[:len(a)] = a
    return out


def _resident_matrix(st, code):
    def read():
        api = _api()
        plen, nv = api.export_size(st.C)
        room = _room(st.case)
        p, i, x = np.zeros(plen, np.int64), np.zeros(room, np.int64), np.zeros(room, NP[code])
        api.matrix_export(st.C, code, p.ctypes.data, i.ctypes.data, x.ctypes.data, plen, nv)
        return {"p": p, "i": i, "x": x}
    return Resident(("p", "i", "x"), read)


def _resident_vector(st, v, code, missing):
    def read():
        api = _api()
        nv = api.vnvals(v)
        i, x = np.zeros(nv, np.int64), np.zeros(nv, NP[code])
        api.vector_extract(v, code, i.ctypes.data, x.ctypes.data, nv)
        dense = np.full(st.case["n"], missing, NP[code])
        dense[i] = x
        return {"x": dense}
    return Resident(("x",), read)


def _resident_batch(st):
    def read():
        p, i, x, nnz = st.batch.result_arrays()
        room = _room(st.case)
        return {"p": p, "i": _padded(i, room), "x": _padded(x, room), "nnz": nnz}
    return Resident(("p", "i", "x", "nnz"), read)


# ---------------------------------------------------------------------------
# what a program holds before the call, and the call
# ---------------------------------------------------------------------------

class State:
    """Handles of one prepared case, freed with it."""

    def __init__(self, case):
        self.case = case
        self.matrices, self.vectors = [], []
        self.batch = None

    def matrix(self, A):
        self.matrices.append(A)
        return A

    def __del__(self):
        try:
            for A in self.matrices:
                _api().free(A)
            for v in self.vectors:
                _api().vfree(v)
            if self.batch is not None:
                self.batch.free()
        except Exception:
            pass


def prepare(case, seed):
    api = _api()
    kind = case["kind"]
    st = State(case)
    if kind == "batch":
        st.batch = B.Batch(_batch(case, seed), semiring("MIN", "PLUS", "fp32"))
        st.batch.tune()
        return st
    n = case["n"]
    if kind in ("triangles", "bfs"):
        p, i = _pattern(case, _generator(seed))
        if kind == "bfs":
            st.A = st.matrix(_import(p, i, _ones(i), BOOL, n))
            st.source = _source(p, seed)
            return st
        row = torch.repeat_interleave(torch.arange(n, device=p.device), p[1:] - p[:-1])
        keys = row * n + i
        Lp, Li = _csr_of_keys(keys[i < row], n, n)
        Up, Ui = _csr_of_keys(keys[i > row], n, n)
        st.L = st.matrix(_import(Lp, Li, _ones(Li), BOOL, n))
        st.U = st.matrix(_import(Up, Ui, _ones(Ui), BOOL, n))
        st.C = st.matrix(api.matrix_new(INT64, n, n))
        return st
    p, i, x, code = _matrix(case, seed)
    if kind == "round_trip":
        pin = torch.cuda.is_available()
        st.host = [t.cpu().pin_memory() if pin else t.cpu() for t in (p, i, x)]
        room = _room(case)                          # every product an entry of its own
        st.out = [torch.zeros(k, dtype=d, pin_memory=pin) for k, d in
                  ((n + 1, torch.int64), (room, torch.int64), (room, torch.float64))]
        return st
    st.A = st.matrix(_import(p, i, x, code, n))
    if kind == "sssp":
        st.source = _source(p, seed)
    else:
        st.C = st.matrix(api.matrix_new(code, n, n))
    return st


def run(st):
    api = _api()
    case = st.case
    kind = case["kind"]
    if kind == "batch":
        st.batch.run()
        return _resident_batch(st)
    n = case["n"]
    if kind == "triangles":
        api.mxm(st.C, st.L, None, "GxB_PLUS_PAIR_INT64", st.L, st.U, "GrB_DESC_ST1")
        return {"triangles": api.reduce(st.C, "GrB_PLUS_MONOID_INT64", INT64),
                "C": _resident_matrix(st, INT64)}
    if kind == "similarity":
        api.mxm(st.C, st.A, None, "GrB_PLUS_TIMES_SEMIRING_FP64", st.A, st.A, "GrB_DESC_ST1")
        return _resident_matrix(st, FP64)
    if kind == "product":
        name, code = PRODUCT[case["semiring"]]
        api.mxm(st.C, None, None, name, st.A, st.A)
        return _resident_matrix(st, code)
    if kind == "round_trip":
        p, i, x = st.host
        cp, ci, cx = st.out
        A = api.matrix_import(FP64, n, n, p.data_ptr(), i.data_ptr(), x.data_ptr(), len(i))
        C = api.matrix_new(FP64, n, n)
        api.mxm(C, None, None, "GrB_PLUS_TIMES_SEMIRING_FP64", A, A)
        api.matrix_export(C, FP64, cp.data_ptr(), ci.data_ptr(), cx.data_ptr(), n + 1, len(ci))
        api.free(A)
        api.free(C)
        return {"p": cp, "i": ci, "x": cx}
    # a traversal's vectors are the caller's until the next one
    while st.vectors:
        api.vfree(st.vectors.pop())
    if kind == "sssp":
        d = api.vector_from([st.source], [0.0], FP32, n)
        st.vectors = [d]
        for _ in range(case["hops"]):
            api.vxm(d, None, "GrB_MIN_FP32", "GrB_MIN_PLUS_SEMIRING_FP32", d, st.A)
        return _resident_vector(st, d, FP32, np.inf)
    q = api.vector_from([st.source], [st.source], INT64, n)
    parent = api.vector_from([st.source], [st.source], INT64, n)
    st.vectors = [q, parent]
    while True:
        # S is symmetric: a level with a large frontier asks every unvisited
        # vertex for its largest frontier neighbour instead
        if case["pull"] and api.vnvals(q) > n // 32:
            api.mxv(q, parent, None, "GxB_MAX_SECONDI_INT64", st.A, q, "GrB_DESC_RSC")
        else:
            api.vxm(q, parent, None, "GxB_ANY_SECONDI_INT64", q, st.A, "GrB_DESC_RSC")
        if api.vnvals(q) == 0:
            break
        api.assign_all(parent, q, None, q, n, "GrB_DESC_S")
    return _resident_vector(st, parent, INT64, -1)


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how close its result has to be
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _product_sizes(n, graph, ef, dmin, dmax):
    """(entries of A, products of A*A, entries of A*A) about."""
    if graph == "er":
        d = (dmin + dmax) / 2
        prod = n * d * d
        return n * d, prod, n * n * (1 - math.exp(-prod / n / n))
    p, i = _rmat(n, ef, _generator(1))
    deg = (p[1:] - p[:-1]).double()
    per_entry = torch.zeros(len(i) + 1, dtype=torch.float64, device=i.device)
    per_entry[1:] = torch.cumsum(deg[i], 0)
    f = per_entry[p[1:]] - per_entry[p[:-1]]                     # products of each row
    # a skewed graph's products meet more often than uniform ones would
    return len(i), float(f.sum()), float((n * (1 - torch.exp(-f / (2 * n)))).sum())


def work(case):
    kind = case["kind"]
    if kind == "batch":
        rows = sum(_batch_sizes(case))                # six entries a row
        return {"bytes": 2 * 4 * rows + 8 * 6 * rows + 8 * 35 * rows, "flops": 2 * 36 * rows}
    n = case["n"]
    if kind == "triangles":
        nnz = case["ef"] * n * 0.95
        # L, U and the mask (L in its own pass) read, C written, 4-byte
        # indices and 8-byte counts
        return {"bytes": 3 * 4 * (n + nnz) + 4 * n + 12 * nnz, "flops": 0}
    if kind == "bfs":
        # every row once, the parents written once
        return {"bytes": 8 * n + 4 * 2 * case["ef"] * n * 0.95 + 8 * n, "flops": 0}
    if kind == "sssp":
        nnz = 2 * case["ef"] * n * 0.95
        # every hop that reaches the graph reads it; the first ones do not
        hops = max(1, case["hops"] - 2)
        return {"bytes": hops * (4 * n + 8 * nnz + 8 * n), "flops": 2 * hops * nnz}
    if kind == "similarity":
        nnz, prod, _ = _product_sizes(n, "rmat", case["ef"], 0, 0)
        return {"bytes": 4 * n + 12 * nnz + 12 * nnz, "flops": 2 * nnz}
    nnz, prod, nnz_c = _product_sizes(n, case.get("graph", "er"), case.get("ef"),
                                      case.get("dmin"), case.get("dmax"))
    size = 4 if case.get("semiring", "").endswith("fp32") else 8
    w = {"bytes": 8 * n + (4 + size) * (nnz + nnz_c), "flops": 2 * prod}
    if kind == "round_trip":
        w["bytes"] += 16 * (n + nnz + nnz_c)        # the int64 arrays of the host
    return w


def tolerance(case):
    """Integers and fp32 minima are the same in any order; floating sums may
    be added in another one."""
    kind = case["kind"]
    name = case.get("semiring", "plus_times_fp64")
    if kind in ("triangles", "bfs", "sssp", "batch") or name == "min_plus_fp32":
        return "exact"
    # sums of up to some hundred terms of either sign: four times what adding
    # them in another order shows
    return {"rel": 4e-7, "max": 1e-4} if name == "plus_times_fp32" else {"rel": 2e-15, "max": 2e-13}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _expand(p, i, x, q, j, y):
    """The products of the CSR matrices (p, i, x) and (q, j, y): for each, the
    row and column in C and the two values."""
    row = torch.repeat_interleave(torch.arange(len(p) - 1, device=p.device), p[1:] - p[:-1])
    length = (q[1:] - q[:-1])[i]
    e = torch.repeat_interleave(torch.arange(len(i), device=p.device), length)
    start = torch.cumsum(length, 0) - length
    at = q[i[e]] + torch.arange(len(e), device=p.device) - start[e]
    return row[e], j[at], x[e], y[at]


def _fold(keys, z, minimum):
    """The values of equal keys folded, in ascending key order."""
    uniq, inverse = torch.unique(keys, return_inverse=True)
    if minimum:
        out = torch.full((len(uniq),), math.inf, dtype=torch.float64, device=z.device)
        return uniq, out.scatter_reduce_(0, inverse, z, "amin")
    return uniq, torch.zeros(len(uniq), dtype=torch.float64, device=z.device).index_add_(
        0, inverse, z)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("triangles", "bfs"):
        return None                                   # whole numbers alone
    if kind == "batch":
        out = []
        for A in _batch(case, seed):
            p, i, x = (torch.from_numpy(t).to(_device()) for t in (A.p, A.i, A.x.astype(np.float64)))
            r, c, a, b = _expand(p, i, x, p, i, x)
            out.append(_fold(r * A.nrows + c, a + b, True)[1].cpu().numpy())
        return {"p": None, "i": None, "x": _padded(np.concatenate(out), _room(case)), "nnz": None}
    n = case["n"]
    p, i, x, _ = _matrix(case, seed)
    x = x.double()
    row = torch.repeat_interleave(torch.arange(n, device=p.device), p[1:] - p[:-1])
    if kind == "sssp":
        d = torch.full((n,), math.inf, dtype=torch.float64, device=p.device)
        d[_source(p, seed)] = 0.0
        for _ in range(case["hops"]):
            d = d.clone().scatter_reduce_(0, i, d[row] + x, "amin")
        return {"x": d.cpu().numpy()}
    if kind == "similarity":
        # the transpose, then the products whose place is in A's pattern
        order = torch.sort(i * n + row)[1]
        tp, ti = _csr_of_keys((i * n + row)[order], n, n)
        r, c, a, b = _expand(p, i, x, tp, ti, x[order])
        keys, pattern = r * n + c, row * n + i
        at = torch.searchsorted(pattern, keys).clamp_(max=len(pattern) - 1)
        hit = pattern[at] == keys
        _, z = _fold(keys[hit], (a * b)[hit], False)
        return {"p": None, "i": None, "x": _padded(z.cpu().numpy(), _room(case))}
    r, c, a, b = _expand(p, i, x, p, i, x)
    minimum = case.get("semiring") == "min_plus_fp32"
    _, z = _fold(r * n + c, a + b if minimum else a * b, minimum)
    return {"p": None, "i": None, "x": _padded(z.cpu().numpy(), _room(case))}
