"""Matching sweep against the oracle at the row lengths where the preference
sort changes its lanes per row (8, 16, 32): rows of exactly the group's size,
one below and one above (queued for the longer sorts), few and many of them,
distinct and tied weights.  Suitor, matching, aggregates and prolongator
values bit for bit (tests/test_gpu_parity.py states the contract)."""
import numpy as np
import pytest
import scipy.sparse as sp

import bootcmatchg_b200 as bc
from oracle import oracle as orc

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def banded(n, half, extra, seed, ties):
    """2 half + 1 entries in most rows; every `extra`-th row coupled to one
    further row (0: none), so some rows are one entry longer."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n - k) for k in range(1, half + 1)])
    j = np.concatenate([np.arange(k, n) for k in range(1, half + 1)])
    if extra:
        e = np.arange(0, n - half - 7, extra)
        i, j = np.concatenate([i, e]), np.concatenate([j, e + half + 5])
    v = -np.ones(i.size) if ties else -rng.uniform(0.5, 2.0, i.size)
    S = sp.coo_matrix((v, (i, j)), shape=(n, n)).tocsr()
    S = S + S.T
    d = np.asarray(abs(S).sum(axis=1)).ravel() + 0.5
    return bc.CsrMatrix.from_scipy((S + sp.diags(d)).tocsr())


def matches_oracle(A, ties):
    from test_gpu_parity import gpu_pair_aggregate
    n = A.n
    w = np.ones(n) if ties else np.random.default_rng(n + 1).uniform(0.5, 1.5, n)
    g, o = gpu_pair_aggregate(A, w), orc.pair_aggregate(A, w)
    np.testing.assert_allclose(g["W"], o["W"], rtol=4 * 2.0 ** -52, atol=0)
    for key in ("suitor", "match", "agg", "p"):
        assert np.array_equal(g[key], o[key]), key
    assert g["nc"] == o["nc"]


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n,half,extra", [(1003, 1, 0), (2049, 2, 3), (65, 3, 0), (1500, 4, 0),
                                          (3001, 3, 2), (777, 7, 0), (1600, 8, 9),
                                          (2000, 5, 4), (900, 15, 3), (500, 20, 0)])
def test_matching_at_group_edges(n, half, extra, ties):
    matches_oracle(banded(n, half, extra, seed=n, ties=ties), ties)


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("half", [4, 8, 15, 16, 31, 32])
def test_matching_of_two_row_populations(half, ties):
    """Short rows with some far longer ones (9, 17, 31, 33, 63 and 65 entries),
    few enough that the mean picks 8 or 16 lanes per row: the long ones are
    all queued, one, two or four entries per lane."""
    short, wide = 40 * half, 3 * half
    A = sp.block_diag([banded(short, 1, 0, half, ties).to_scipy(),
                       banded(wide, half, 0, half + 1, ties).to_scipy()]).tocsr()
    assert A.nnz <= 11 * A.shape[0]
    matches_oracle(bc.CsrMatrix.from_scipy(A), ties)
