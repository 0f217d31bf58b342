"""Smoother sweeps of one level against a plain numpy sweep, at the edges of
the row passes: column slices of every batch remainder, slices cut by the last
row, offset slices inside a copy of column slices, constant-coefficient
stencils of the widths kernels are built for and of others, with and without
missing entries, and levels small enough for one thread-block cluster
(distributed or replicated iterate).

One sweep (k = 1) runs the row pass, several run the cluster kernel where the
level fits one.  Bound per row and sweep: a sum of m products in any order is
within (m + 2) eps of the sum of their magnitudes, the division and the two
additions within 3 eps of theirs; the errors of earlier sweeps pass through
|I - D^-1 A|, whose row sums are at most 2 for the l1 diagonal.
"""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import bootcmatchg_b200 as bc
import workloads as wl
from bootcmatchg_b200._lib import check, lib
from helpers import c1_params, random_sym_graph

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def constant_stencil(offsets, n, seed):
    """One coefficient per offset, some entries left out at random: a uniform
    copy whose rows have arbitrary masks."""
    rng = np.random.default_rng(seed)
    r = np.concatenate([np.arange(n - o) for o in offsets])
    c = np.concatenate([np.arange(o, n) for o in offsets])
    v = np.concatenate([np.full(n - o, -0.3 - 0.1 * k) for k, o in enumerate(offsets)])
    keep = rng.uniform(size=r.size) < 0.97
    S = sp.coo_matrix((v[keep], (r[keep], c[keep])), shape=(n, n)).tocsr()
    return bc.CsrMatrix.from_scipy((S + S.T + sp.identity(n) * 9.7).tocsr())


def banded_and_random(n):
    """A 5-point band on the first half of the rows, random columns on the rest."""
    g = random_sym_graph(n // 2, 9, seed=5, int_weights=False).to_scipy()
    m = n - n // 2
    band = sp.diags([-1.0, -1.0, 4.0, -1.0, -1.0], [-7, -1, 0, 1, 7], shape=(m, m))
    return bc.CsrMatrix.from_scipy(sp.block_diag([band, g]).tocsr())


CASES = {
    "rand_33_w3": lambda: random_sym_graph(33, 2, seed=1, int_weights=False),
    "rand_1000_w8": lambda: random_sym_graph(1000, 4, seed=2, int_weights=False),
    "rand_1025_w20": lambda: random_sym_graph(1025, 12, seed=3, int_weights=False),
    "rand_2500_w50": lambda: random_sym_graph(2500, 36, seed=4, int_weights=False),
    "rand_40007_w24": lambda: random_sym_graph(40007, 14, seed=6, int_weights=False),
    "band_and_rand_3011": lambda: banded_and_random(3011),
    "rgg_5003": lambda: wl.rgg(5003, seed=9),
    "poisson7_13x11x9": lambda: wl.poisson(7, 13, 11, 9),
    "poisson27_31": lambda: wl.poisson(27, 31, 31, 31),
    "poisson27_70x33x5": lambda: wl.poisson(27, 70, 33, 5),
    "poisson5_257x129": lambda: wl.poisson(5, 257, 129),
    "const_w7_no_runs": lambda: constant_stencil([2, 5, 40], 9001, 1),
    "const_w31": lambda: constant_stencil(list(range(1, 16)), 20011, 2),
    "const_w27_no_runs": lambda: constant_stencil([1, 2, 3, 5, 8, 13, 21, 34, 55, 89, 144, 233,
                                                   377], 30000, 3),
}


@pytest.mark.parametrize("precision", [bc.PREC_FP64, bc.PREC_MIXED])
@pytest.mark.parametrize("case", sorted(CASES))
def test_sweeps_match_numpy(case, precision):
    A = CASES[case]()
    mixed = precision == bc.PREC_MIXED
    eps, dt = (2.0 ** -24, np.float32) if mixed else (2.0 ** -53, np.float64)
    f = wl.vector(1, 1, A.n).astype(dt)
    u0 = wl.vector(2, 2, A.n).astype(dt)
    with bc.Handle(A, c1_params(), bc.Extensions(precision=precision)) as h:
        M = h.level(0, 0).M.astype(dt).astype(np.float64)
        S = sp.csr_matrix((np.asarray(A.val).astype(dt).astype(np.float64), A.col, A.row),
                          shape=(A.n, A.n))
        m = int(np.diff(S.indptr).max())
        for k in (1, 2, 5):
            fd, ud = torch.from_numpy(f).cuda(), torch.from_numpy(u0).cuda()
            check(lib.bcmg_level_relax(h.ptr, 0, 0, C.c_void_p(fd.data_ptr()),
                                       C.c_void_p(ud.data_ptr()), k), "level_relax")
            u, err = u0.astype(np.float64), np.zeros(A.n)
            f64 = f.astype(np.float64)
            for _ in range(k):
                mag = (abs(S) @ abs(u) + abs(f64)) / abs(M) + abs(u)
                err = err + abs(S) @ err / abs(M) + (m + 5) * 1.01 * eps * mag
                u = u + (f64 - S @ u) / M
            assert np.all(abs(ud.cpu().numpy() - u) <= err), (case, k)
