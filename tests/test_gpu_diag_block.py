"""Diagonal blocks factored and inverted in one launch (diag_block_kernel), through
moao_dense_potrf_inv: one column past a leaf, uneven halves, remainders of the 32-wide
tiles, the widest block, odd leading dimensions (8-byte loads); and through the FP64
reconstructor with one and eight CTAs beside other work, which must give the same bits.

Tolerances: |L L^T - A| <= (n + 1) eps sqrt(a_ii a_jj) elementwise for a Cholesky factor
in FP64, four times that for the reciprocal square roots. The blocked inverse, as the
substitution of the oracle, is good to 4 n eps kappa(L) of its norm; both together 8."""
import ctypes as C

import numpy as np
import pytest
import scipy.linalg as sl

import moao_b200 as M
from moao_b200._lib import lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def factor(ctx, A, ld):
    import torch
    n = A.shape[0]
    buf = np.full((n, ld), 7.0)
    buf[:, :n] = A.T
    a = torch.from_numpy(buf).cuda()
    x = torch.full((n, ld), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info = C.c_int(-1)
    st = lib().moao_dense_potrf_inv(ctx.handle, n, a.data_ptr(), ld, x.data_ptr(), ld, C.byref(info))
    return st, info.value, a.cpu().numpy(), x.cpu().numpy()


def spd(n):
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n + 3))
    s = 2.0 ** rng.integers(-8, 9, n)
    return s[:, None] * (B @ B.T / n + 0.05 * np.eye(n)) * s[None, :]


@pytest.mark.parametrize("n,pad", [(65, 0), (65, 1), (95, 0), (129, 0), (161, 2), (192, 3), (255, 0), (257, 0),
                                   (640, 0), (1023, 0), (1024, 0), (1024, 5), (1900, 0), (2048, 0), (2100, 0)])
def test_factor_and_inverse(ctx, n, pad):
    A = spd(n)
    st, info, a, x = factor(ctx, A, n + pad)
    assert st == 0 and info == 0
    L, X = np.tril(a[:, :n].T), x[:, :n].T
    d = np.sqrt(np.diag(A))
    assert np.max(np.abs(L @ L.T - A) / np.outer(d, d)) <= 4 * (n + 1) * EPS
    want = sl.solve_triangular(L, np.eye(n), lower=True)
    kappa = np.linalg.norm(want) * np.linalg.norm(L)
    assert np.linalg.norm(X - want) <= 8 * n * EPS * kappa * np.linalg.norm(want)
    assert np.array_equal(np.triu(X, 1), np.zeros((n, n)))
    assert np.array_equal(np.triu(a[:, :n].T, 1), np.triu(A, 1))
    assert np.all(a[:, n:] == 7.0) and np.all(x[:, n:] == 7.0)


@pytest.mark.parametrize("n,bad", [(65, 65), (300, 64), (300, 192), (1024, 513), (1024, 1024), (2048, 1500)])
def test_first_bad_pivot_is_reported(ctx, n, bad):
    A = spd(n)
    A[bad - 1, bad - 1] = -1.0
    st, info, _, _ = factor(ctx, A, n)
    assert st == 2 and info == bad


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_number_of_ctas_does_not_change_R(prec, built, cuda):
    import torch
    n, m = 6 * 1024 + 100, 300
    x = torch.linspace(0, 60, n, dtype=torch.float64, device="cuda")
    s = torch.exp(-(x[:, None] - x[None, :]).abs()) + 0.01 * torch.eye(n, dtype=x.dtype, device="cuda")
    t = torch.exp(-(x[None, :m] - x[:, None]).abs())
    out = []
    for sms in (1, 8, 0):  # CTAs beside the update; none beside it
        ctx = M.Context(0)
        ctx.set_lookahead(sms)
        Cmm, Ctm = torch.tril(s).T.contiguous(), t.clone()
        M.reconstructor(n, m, Cmm, n, Ctm, m, 1, prec=prec, ctx=ctx)
        out.append(Ctm)
        ctx.close()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
