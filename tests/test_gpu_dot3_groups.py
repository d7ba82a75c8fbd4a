"""Counting dot products (PLUS_PAIR) with fewer columns than the grouped path's
bitmap once needed: masks on either side of the entries from which they are
grouped, key rows for the hash table and the bitmap, and one-word rows.
Checked against the oracle."""

import numpy as np
import pytest

from graphblas_b200 import workloads as W
from tests.helpers import assert_exact, random_csr

pytestmark = pytest.mark.gpu
LENGTHS = [0, 1, 7, 40, 255, 256, 257, 511, 512, 513, 900, 1500]


def rows_of(nrows, ncols, seed):
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(ncols, min(int(k), ncols), replace=False))
            for k in rng.choice(LENGTHS, nrows)]
    p = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return W.Csr(nrows, ncols, p, np.concatenate(rows).astype(np.int64), None)


@pytest.mark.parametrize("tname", ["int64", "int32"])
@pytest.mark.parametrize("density", [0.3, 1.0])
@pytest.mark.parametrize("k", [33, 3000, 32735, 32736])
def test_grouped_counts_few_columns(gpu, oracle, tname, density, k):
    gb = gpu
    tc = gb.TYPES[tname]
    m, n = 360, 370                       # 40 thousand mask entries, and 133 thousand
    A, B = rows_of(m, k, 1), rows_of(n, k, 2)
    M = random_csr(m, n, density, 3, np.bool_)
    M.x = None
    dA, dB, dM = (gb.DMatrix.upload(X, "bool") for X in (A, B, M))
    C = gb.dot3(dM, dA, dB, gb.semiring("PLUS", "PAIR", tname))
    total = int(gb.reduce(C, "PLUS", gb.NP_OF[tc]))
    got = C.download(prune=True)
    want = oracle.dot3(m, n, (A.p, A.i, None, 1), (B.p, B.i, None, 1), (M.p, M.i, None, 1),
                       "PLUS", "PAIR", tc)
    assert_exact(got, want, tname)
    assert total == int(np.sum(want[2], dtype=np.int64))
    for d in (dA, dB, dM, C):
        d.free()
