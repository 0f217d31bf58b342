"""Calls on a caller's stream see what the caller's stream copies wrote.

Each call's device vectors are overwritten by asynchronous device-to-device
copies on the handle's stream directly before the call, with no
synchronisation between; the result has the bits of the same call on vectors
that were complete before it.  The blocks are large (7-point Poisson 96^3, 32
columns where batched: copies of 113 to 226 MB take tens of microseconds), so
a first kernel that does not wait for the copies reads what was there before.
"""
import ctypes as C

import numpy as np
import pytest

import bootcmatchg_b200 as bc
import workloads as wl
from bootcmatchg_b200._lib import check, lib
from helpers import c1_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W = 32


@pytest.fixture(scope="module", params=[bc.PREC_FP64, bc.PREC_MIXED], ids=["fp64", "mixed"])
def bound(request):
    """A handle bound to a torch stream, and that stream."""
    mixed = request.param == bc.PREC_MIXED
    stream = torch.cuda.Stream()
    A = wl.poisson(7, 96, 96, 96)
    ext = bc.Extensions(precision=request.param, replace_every=10 if mixed else 0, autotune=0,
                        stream=stream.cuda_stream)
    with bc.Handle(A, c1_params(), ext) as h:
        yield h, stream, torch.float32 if mixed else torch.float64


def block(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, dtype=dtype, device="cuda", generator=g)


def same_after_copies(stream, call, vin, vout):
    """call(vin', vout') with vin' and vout' complete before it, then written
    by stream copies just before it: equal bits in vout'."""
    a, b = vin.clone(), vout.clone()
    torch.cuda.synchronize()
    call(a, b)
    torch.cuda.synchronize()
    for _ in range(3):
        c, d = torch.full_like(vin, 7.0), torch.full_like(vout, -5.0)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            c.copy_(vin, non_blocking=True)
            d.copy_(vout, non_blocking=True)
        call(c, d)
        torch.cuda.synchronize()
        assert torch.equal(b, d)


def ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("k", [1, 2, 5])
def test_level_relax(bound, k):
    h, stream, dt = bound
    for level in (0, 1):
        n = h.level(0, level).n
        same_after_copies(
            stream, lambda f, u: check(lib.bcmg_level_relax(h.ptr, 0, level, ptr(f), ptr(u), k),
                                       "level_relax"), block(n, dt, 1), block(n, dt, 2))


@pytest.mark.parametrize("k", [1, 2, 5])
def test_level_relax_batch(bound, k):
    h, stream, dt = bound
    for level in (0, 1):
        n = h.level(0, level).n * W
        same_after_copies(
            stream,
            lambda f, u: check(lib.bcmg_level_relax_batch(h.ptr, 0, level, W, ptr(f), ptr(u), k),
                               "level_relax_batch"), block(n, dt, 3), block(n, dt, 4))


def test_precond_apply(bound):
    h, stream, _ = bound
    same_after_copies(stream, lambda r, z: h.precond_apply_device(r.data_ptr(), z.data_ptr()),
                      block(h.n, torch.float64, 5), block(h.n, torch.float64, 6))
    n = h.n
    same_after_copies(
        stream,
        lambda r, z: h.precond_apply_batch_device(W, r.data_ptr(), n, z.data_ptr(), n),
        block(n * W, torch.float64, 7), block(n * W, torch.float64, 8))


@pytest.mark.parametrize("call", ["bcmg_k_relax", "bcmg_k_relax_noalloc"])
@pytest.mark.parametrize("k", [1, 2])
def test_single_step_relax(call, k):
    A = wl.poisson(7, 96, 96, 96)
    stream = torch.cuda.Stream()
    m = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.row, A.col, A.val)]
    d = torch.full((A.n,), 13.0, dtype=torch.float64, device="cuda")
    same_after_copies(
        stream,
        lambda f, u: check(getattr(lib, call)(A.n, A.nnz, *map(ptr, m), ptr(d), ptr(f), ptr(u), k,
                                              C.c_void_p(stream.cuda_stream)), call),
        block(A.n, torch.float64, 13), block(A.n, torch.float64, 14))


def test_solves(bound):
    h, stream, _ = bound
    n = h.n
    same_after_copies(stream, lambda b, x: h.solve_device(b.data_ptr(), x.data_ptr()),
                      block(n, torch.float64, 9), block(n, torch.float64, 10))
    same_after_copies(
        stream, lambda b, x: h.solve_batch_device(W, b.data_ptr(), n, x.data_ptr(), n),
        block(n * W, torch.float64, 11), block(n * W, torch.float64, 12))
