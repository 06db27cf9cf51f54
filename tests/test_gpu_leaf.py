"""The leaf factorisation with inverse (leaf_f64.cuh) through moao_dense_potrf_inv
at the sizes where it can go wrong: one column, around its 16-wide sub-blocks,
around its 64-wide limit (two leaves), and with a padded leading dimension.

Tolerances: a Cholesky factor computed in FP64 satisfies
|L L^T - A| <= (n + 1) eps |L| |L^T| elementwise, at most (n + 1) eps sqrt(a_ii a_jj);
four times that covers the reciprocal square roots (a few eps per pivot instead
of half). The inverse of the computed factor satisfies ||X L - I||_F <=
4 n eps ||X||_F ||L||_F."""
import ctypes as C

import numpy as np
import pytest

import moao_b200 as M
from moao_b200._lib import lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
SIZES = [1, 2, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 80, 128]


def spd(n, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((n, n + 3))
    s = 2.0 ** rng.integers(-8, 9, n)  # rows and columns at uneven scales
    return s[:, None] * (B @ B.T / n + 0.05 * np.eye(n)) * s[None, :]


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


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("pad", [0, 3])
def test_factor_and_inverse(ctx, n, pad):
    A = spd(n, n)
    st, info, a, x = factor(ctx, A, n + pad)
    assert st == 0 and info == 0
    L, X = np.tril(a[:, :n].T), x[:, :n].T
    d = np.sqrt(np.diag(A))
    assert np.max(np.abs(L @ L.T - A) / np.outer(d, d)) <= 4 * (n + 1) * EPS
    assert np.linalg.norm(X @ L - np.eye(n)) <= 4 * n * EPS * np.linalg.norm(X) * np.linalg.norm(L)
    assert np.array_equal(np.triu(X, 1), np.zeros((n, n)))
    # the upper triangle and the padding are left alone
    assert np.array_equal(np.triu(a[:, :n].T, 1), np.triu(A, 1))
    assert np.all(a[:, n:] == 7.0) and np.all(x[:, n:] == 7.0)


@pytest.mark.parametrize("n,bad", [(1, 1), (40, 1), (40, 16), (40, 17), (64, 64), (100, 65), (100, 100)])
def test_first_bad_pivot_is_reported(ctx, n, bad):
    A = spd(n, 3 * n)
    A[bad - 1, bad - 1] = -1.0
    st, info, _, _ = factor(ctx, A, n)
    assert st == 2 and info == bad
    st, info, _, _ = factor(ctx, spd(n, 5), n)
    assert st == 0 and info == 0
