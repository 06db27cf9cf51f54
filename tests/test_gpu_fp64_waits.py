"""The FP64 path's bounded device waits, made to run out by a limit of one poll (the
kernels give up, end and leave the context usable). A residue product whose waits ran out
is computed by the FP64 tensor cores, tile range by tile range: its bound is that of
test_gpu_crt64.py, which covers both. A diagonal block whose barrier ran out ends its call
with MOAO_ERR_TIMEOUT."""
import ctypes as C

import numpy as np
import pytest

import moao_b200 as M
from moao_b200._lib import check, lib
from test_gpu_crt64 import check_close, product, values
from test_gpu_memory import rec, rel, system

pytestmark = pytest.mark.gpu


@pytest.fixture
def own(built, cuda):
    c = M.Context(0)
    yield c
    c.close()


def waits(ctx, product_polls, barrier_polls):
    check(lib().moao_debug_fp64_waits(ctx.handle, product_polls, barrier_polls), "waits")


@pytest.mark.parametrize("form,lower", [(0, 0), (0, 1), (1, 0), (2, 0)])
@pytest.mark.parametrize("tiles", [0, 2])
def test_products(own, form, lower, tiles):
    rng = np.random.default_rng(form)
    m = n = 700
    k = 700 if form == 2 else 4000
    A, Bt = values(rng, m, k), values(rng, n, k)
    if form == 2:
        Bt = np.tril(Bt) + np.tril(Bt, -1).T
    beta = 0.0 if form == 2 else 1.0
    C0 = rng.standard_normal((m, n)) * beta
    args = (form, lower, A, {0: Bt, 1: Bt.T, 2: np.tril(Bt)}[form], 1.0, beta, C0)
    plain = product(own, *args)
    waits(own, 1, 0)
    check(lib().moao_debug_limits(own.handle, 0, 1 if tiles else 0, tiles), "limits")
    got = product(own, *args)
    low = np.tril(np.ones((m, n), bool)) if lower else np.ones((m, n), bool)
    check_close(got, A, Bt, 1.0, beta, C0, low, sym=form == 2)
    assert np.array_equal(got[~low], C0[~low])
    assert not np.array_equal(got, plain)  # it did run out
    waits(own, 0, 0)
    check(lib().moao_debug_limits(own.handle, 0, 0, 0), "limits")
    assert np.array_equal(product(own, *args), plain)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [130, 2500])
def test_diagonal_block(own, prec, n):
    C0, T0, R = system(n, 100)
    waits(own, 0, 1)
    with pytest.raises(M.MoaoError) as e:
        rec(own, n, 100, C0, T0, prec)
    assert e.value.name == "MOAO_ERR_TIMEOUT"
    waits(own, 0, 0)
    assert rel(rec(own, n, 100, C0, T0, prec), R) <= (1e-10 if prec == "fp64" else 1e-5)


def test_dense_potrf_inv(own):
    import torch
    n = 200
    A0, _, _ = system(n, 1)
    A, D, info = A0.clone(), torch.zeros_like(A0), C.c_int32()
    waits(own, 0, 1)

    def run():
        A.copy_(A0)
        torch.cuda.synchronize()
        return lib().moao_dense_potrf_inv(own.handle, n, A.data_ptr(), n, D.data_ptr(), n, C.byref(info))

    with pytest.raises(M.MoaoError) as e:
        check(run(), "potrf")
    assert e.value.name == "MOAO_ERR_TIMEOUT"
    waits(own, 0, 0)
    check(run(), "potrf")
    L = torch.linalg.cholesky(A0)
    assert rel(torch.tril(A.T), L) <= 1e-12
