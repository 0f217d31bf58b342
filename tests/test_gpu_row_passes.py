"""Smoother sweeps of one level against a plain numpy sweep, at the edges of
the row passes: column slices of every batch remainder, slices cut by the last
row, offset slices inside a copy of column slices, stencils of varying and of
constant coefficients, of the widths kernels are built for and of others, with
and without missing entries, constant ones with some slices that are not, and
levels small enough for one thread-block cluster (distributed or replicated
iterate).  Each case names the row pass it is for, and is checked to run it.

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
from helpers import c1_params, random_sym_graph, varying_stencil

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


def partly_constant(width, n, seed, spoiled):
    """A constant stencil of `width` entries per row (an even width: one offset
    without its mirror), except in the last `spoiled` whole slices of 32 rows:
    every other of those has another value on its diagonal, the rest, in each
    row, one entry moved to a random column of those slices."""
    off = {5: [1, 7], 7: [1, 6, 30], 27: [1, 8, 9, 10, 71, 72, 73, 80, 81, 82, 89, 90, 91]}
    off = off.get(width, list(range(1, (width + 1) // 2)))
    d = {o: -0.25 - 0.03125 * i for i, o in enumerate(off)}
    diags = {0: 9.0, **d, **{-o: v for o, v in d.items()}}
    if len(diags) < width:
        diags[max(off) + 5] = -0.75
    S = sp.diags(list(diags.values()), list(diags), shape=(n, n)).tolil()
    rng = np.random.default_rng(seed)
    s1 = n // 32
    for t, s in enumerate(range(s1 - spoiled, s1)):
        r = np.arange(32 * s, 32 * s + 32)
        if t % 2:
            S[r, r] = 9.5 + 0.25 * t
        else:
            S[r, r - 1] = 0.0
            S[r, rng.integers(32 * (s1 - spoiled), 32 * s1, 32)] = -0.125
            S[r, r] = 9.0
    return bc.CsrMatrix.from_scipy(S.tocsr())


BOTH, FP32, NONE = (False, True), (True,), ()  # mixed or not
# name: (row pass, uniform slices beside others, precisions with a cluster, matrix)
CASES = {
    "rand_33_w3": ("columns", False, BOTH,
                   lambda: random_sym_graph(33, 2, seed=1, int_weights=False)),
    "rand_1000_w8": ("columns", False, BOTH,
                     lambda: random_sym_graph(1000, 4, seed=2, int_weights=False)),
    "rand_1025_w20": ("columns", False, BOTH,
                      lambda: random_sym_graph(1025, 12, seed=3, int_weights=False)),
    "rand_2500_w50": ("columns", False, FP32,
                      lambda: random_sym_graph(2500, 36, seed=4, int_weights=False)),
    "rand_40007_w24": ("columns", False, NONE,
                       lambda: random_sym_graph(40007, 14, seed=6, int_weights=False)),
    "band_and_rand_3011": ("columns", False, BOTH, lambda: banded_and_random(3011)),
    "rgg_5003": ("columns", False, FP32, lambda: wl.rgg(5003, seed=9)),
    "poisson7_13x11x9": ("uniform", False, BOTH, lambda: wl.poisson(7, 13, 11, 9)),
    "poisson27_31": ("uniform", False, NONE, lambda: wl.poisson(27, 31, 31, 31)),
    # (its mean slice is 24 slots wide, a width no slice has: not seen as constant)
    "poisson27_70x33x5": ("staged", False, NONE, lambda: wl.poisson(27, 70, 33, 5)),
    "poisson27_66x33x40": ("uniform", False, NONE, lambda: wl.poisson(27, 66, 33, 40)),
    "poisson5_257x129": ("uniform", False, NONE, lambda: wl.poisson(5, 257, 129)),
    "const_w7_no_runs": ("uniform", False, BOTH, lambda: constant_stencil([2, 5, 40], 9001, 1)),
    "const_w31": ("uniform", False, NONE,
                  lambda: constant_stencil(list(range(1, 16)), 20011, 2)),
    "const_w27_no_runs": ("uniform", False, NONE,
                          lambda: constant_stencil([1, 2, 3, 5, 8, 13, 21, 34, 55, 89, 144, 233,
                                                    377], 30000, 3)),
    "vary27_33x31x29": ("staged", False, NONE, lambda: varying_stencil(27, 33, 31, 29, 11)),
    "vary27_15x16x16": ("staged", False, BOTH, lambda: varying_stencil(27, 15, 16, 16, 12)),
    "vary27_ints_33x31x29": ("staged", False, NONE,
                             lambda: varying_stencil(27, 33, 31, 29, 13, ints=True)),
    "vary7_41x39x37": ("staged", False, NONE, lambda: varying_stencil(7, 41, 39, 37, 14)),
    "vary7_13x11x9": ("staged", False, BOTH, lambda: varying_stencil(7, 13, 11, 9, 15)),
    "vary7_ints_41x39x37": ("staged", False, NONE,
                            lambda: varying_stencil(7, 41, 39, 37, 16, ints=True)),
    "vary5_130x127": ("staged", False, NONE, lambda: varying_stencil(5, 130, 127, 1, 17)),
}
for w in (5, 7, 27, 31, 32):
    CASES[f"part_w{w}_3010"] = ("uniform", True, BOTH,
                                lambda w=w: partly_constant(w, 3010, w, 12))
    CASES[f"part_w{w}_20021"] = ("uniform", True, NONE,
                                 lambda w=w: partly_constant(w, 20021, w, 90))
# 100 slices: constant from three quarters of them on
CASES["part_w7_three_quarters"] = ("uniform", True, BOTH, lambda: partly_constant(7, 3200, 5, 25))
CASES["part_w7_below"] = ("staged", False, BOTH, lambda: partly_constant(7, 3200, 5, 26))


@pytest.mark.parametrize("precision", [bc.PREC_FP64, bc.PREC_MIXED])
@pytest.mark.parametrize("case", sorted(CASES))
def test_sweeps_match_numpy(case, precision):
    rows, partly, cluster, matrix = CASES[case]
    A = matrix()
    mixed = precision == bc.PREC_MIXED
    with bc.Handle(A, c1_params(), bc.Extensions(precision=precision)) as h:
        got = h.level_pass(0, 0)
        assert got["pass"] == rows, got
        assert (got["cluster_ctas"] > 0) == (mixed in cluster), got
        if rows == "uniform":
            assert (got["uniform_slices"] < (A.n + 31) // 32) == partly, got
        else:
            assert got["uniform_slices"] == got["masked_slices"] == 0
        val = np.asarray(A.val).astype(np.float32 if mixed else np.float64)
        sweeps_match(h, 0, A, val, mixed, case)


@pytest.mark.parametrize("storage", [bc.STORE_BF16, bc.STORE_FP16])
@pytest.mark.parametrize("stencil,dims,level,cluster",
                         [(27, (96, 96, 96), 3, False), (7, (48, 48, 48), 1, False),
                          (7, (48, 48, 48), 3, True), (5, (300, 200), 1, True)])
def test_rounded_uniform_coarse_level(stencil, dims, level, cluster, storage):
    """A constant-coefficient coarse level whose values are rounded to 16 bits:
    the coefficients in the kernel's parameters are the rounded ones."""
    A = wl.poisson(stencil, *dims)
    ext = bc.Extensions(precision=bc.PREC_MIXED, coarse_storage=storage, replace_every=10)
    with bc.Handle(A, c1_params(), ext) as h:
        got = h.level_pass(0, level)
        assert got["pass"] == "uniform" and (got["cluster_ctas"] > 0) == cluster, got
        M = h.level(0, level).A
        dt = torch.bfloat16 if storage == bc.STORE_BF16 else torch.float16
        val = torch.from_numpy(M.val).to(dt).double().numpy()
        assert not np.array_equal(val, M.val)
        sweeps_match(h, level, M, val, True, stencil)


def sweeps_match(h, level, A, val, mixed, case):
    """1, 2 and 5 sweeps of the level (matrix A's pattern, values val)."""
    eps, dt = (2.0 ** -24, np.float32) if mixed else (2.0 ** -53, np.float64)
    f = wl.vector(1, 1, A.n).astype(dt)
    u0 = wl.vector(2, 2, A.n).astype(dt)
    M = h.level(0, level).M.astype(dt).astype(np.float64)
    S = sp.csr_matrix((val.astype(np.float64), A.col, A.row), shape=(A.n, A.n))
    m = int(np.diff(S.indptr).max())
    for k in (1, 2, 5):
        fd, ud = torch.from_numpy(f).cuda(), torch.from_numpy(u0).cuda()
        check(lib.bcmg_level_relax(h.ptr, 0, level, C.c_void_p(fd.data_ptr()),
                                   C.c_void_p(ud.data_ptr()), k), "level_relax")
        u, err = u0.astype(np.float64), np.zeros(A.n)
        f64 = f.astype(np.float64)
        for _ in range(k):
            mag = (abs(S) @ abs(u) + abs(f64)) / abs(M) + abs(u)
            err = err + abs(S) @ err / abs(M) + (m + 5) * 1.01 * eps * mag
            u = u + (f64 - S @ u) / M
        assert np.all(abs(ud.cpu().numpy() - u) <= err), (case, k)
