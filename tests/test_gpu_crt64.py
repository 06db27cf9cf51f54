"""FP64 products as int8 residue products (crt_f64.cu), at the sizes where they
can go wrong: around the 128 x 256 tiles, the 32-wide conversion tiles and the
128-wide K blocks, one row, more than one band of tiles, K past 2^15 (fewer
operand bits), and the forms they take (transposed and plain second operand,
lower triangle only, symmetric operand in its lower triangle).

Oracle: the products of the operands' exact integers (Python integers, small
sizes) or torch's FP64 product on the same device.

Tolerance. With a symmetric second operand S, column k of A is first scaled by
2^s_k and row k of S by 2^-s_k, s_k half the exponent of S(k, k) rounded down;
with a_r, b_c the rows' maxima (scaled), every element is rounded to `bits` bits
of its row's maximum (57 for K <= 1,024, at least 53 for K < 2^17), so it differs
by at most 2^-bits of that maximum, the reconstruction is good to 2^-69 of the moduli's product
(at most 2^-bits of K a_r b_c again), and the update of C adds three roundings:
  |C - exact| <= |alpha| 2^(1 - bits) K a_r b_c + 4 eps (|alpha P| + |beta C|).
Torch's own product is off by at most K eps |A| |B|^T; the bound is the sum."""
import ctypes as C  # noqa: F401
import math

import numpy as np
import pytest

import moao_b200 as M
from moao_b200._lib import check, lib

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
LOG2M = sum(math.log2(m) for m in (256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211,
                                   199, 197, 193))


def bits(K):
    return min(57, math.floor((LOG2M - 1 - math.log2(K) - 1e-6) / 2))


def gpu(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def values(rng, rows, cols):
    """Rows at uneven scales, entries over a few binary orders."""
    return (rng.standard_normal((rows, cols)) * 2.0 ** rng.integers(-6, 3, (rows, cols)) *
            2.0 ** rng.integers(-30, 31, (rows, 1)))


def product(ctx, form, lower, A, B, alpha, beta, C0):
    """Column-major device copies (as transposes); returns C."""
    import torch
    m, k = A.shape
    n = B.shape[0] if form == 0 else B.shape[1]
    a, b, c = gpu(A.T), gpu(B.T), gpu(C0.T)
    torch.cuda.synchronize()
    check(lib().moao_debug_crt64(ctx.handle, form, lower, m, n, k, alpha, a.data_ptr(), m, b.data_ptr(),
                                 b.shape[1], beta, c.data_ptr(), m), "crt64")
    ctx.synchronize()
    return c.cpu().numpy().T


def row_maxima(A, Bt, balanced):
    """Row maxima of A and Bt after the balance along K."""
    s = np.zeros(A.shape[1])
    if balanced:
        s = np.floor((np.frexp(np.diag(Bt))[1] - 1) / 2)
    return (np.abs(A) * 2.0 ** s).max(1)[:, None], (np.abs(Bt) * 2.0 ** -s).max(1)[None, :]


def check_close(got, A, Bt, alpha, beta, C0, mask=None, sym=False):
    """Bt: N x K, C = alpha A Bt^T + beta C0."""
    K = A.shape[1]
    P = (gpu(A) @ gpu(Bt).T).cpu().numpy()
    absP = (gpu(np.abs(A)) @ gpu(np.abs(Bt)).T).cpu().numpy()
    want = alpha * P + beta * C0
    a, b = row_maxima(A, Bt, sym)
    lim = abs(alpha) * (2.0 ** (1 - bits(K)) * K * a * b + K * EPS * absP) + 4 * EPS * (np.abs(alpha * P) + np.abs(beta * C0))
    bad = np.abs(got - want) > lim
    if mask is not None:
        bad &= mask
    assert not bad.any(), np.argwhere(bad)[:5]


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 257, 33), (127, 255, 127), (128, 256, 128), (129, 257, 129),
                                   (300, 500, 1024), (2200, 300, 200), (64, 64, 1025), (40, 50, 40000)])
@pytest.mark.parametrize("form", [0, 1])
def test_products(ctx, m, n, k, form):
    rng = np.random.default_rng(m + n + k)
    A, Bt = values(rng, m, k), values(rng, n, k)
    C0 = rng.standard_normal((m, n))
    got = product(ctx, form, 0, A, Bt if form == 0 else Bt.T, -1.0, 1.0, C0)
    check_close(got, A, Bt, -1.0, 1.0, C0)
    got = product(ctx, form, 0, A, Bt if form == 0 else Bt.T, 0.75, 0.0, np.full((m, n), np.nan))
    check_close(got, A, Bt, 0.75, 0.0, np.zeros((m, n)))


def test_exact_integers(ctx):
    """Integer operands of 25 bits against Python integers, the largest sums included."""
    rng = np.random.default_rng(5)
    A = rng.integers(-2 ** 25, 2 ** 25 + 1, (70, 300)).astype(np.float64)
    B = rng.integers(-2 ** 25, 2 ** 25 + 1, (90, 300)).astype(np.float64)
    A[0], B[0] = 2.0 ** 25, 2.0 ** 25 - 1
    A[1], B[1] = -2.0 ** 25, -1.0
    got = product(ctx, 0, 0, A, B, 1.0, 0.0, np.zeros((70, 90)))
    want = A.astype(np.int64).astype(object) @ B.astype(np.int64).astype(object).T
    w = want.astype(np.float64)
    a, b = row_maxima(A, B, False)
    lim = 2.0 ** (1 - bits(300)) * 300 * a * b + 4 * EPS * np.abs(w)
    assert np.all(np.abs(got - w) <= lim)


@pytest.mark.parametrize("n,k", [(100, 70), (257, 128), (700, 1024)])
def test_lower(ctx, n, k):
    rng = np.random.default_rng(n)
    A = values(rng, n, k)
    C0 = rng.standard_normal((n, n))
    got = product(ctx, 0, 1, A, A, -1.0, 1.0, C0)
    low = np.tril(np.ones((n, n), bool))
    check_close(got, A, A, -1.0, 1.0, C0, low)
    assert np.array_equal(got[~low], C0[~low])


@pytest.mark.parametrize("m,n", [(5, 33), (130, 300), (300, 1111)])
def test_symmetric(ctx, m, n):
    rng = np.random.default_rng(n)
    A = values(rng, m, n)
    S = values(rng, n, n)
    S = np.tril(S) + np.tril(S, -1).T
    got = product(ctx, 2, 0, A, np.tril(S) + np.triu(np.full((n, n), np.nan), 1), 1.0, 0.0,
                  np.zeros((m, n)))
    check_close(got, A, S, 1.0, 0.0, np.zeros((m, n)), sym=True)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e290, 1e-300, 5e-324])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_guard_takes_the_fp64_path(ctx, value, form):
    """A non-finite or extreme operand: what the FP64 tensor cores give, every
    other row unaffected."""
    rng = np.random.default_rng(11)
    m, n = 150, 333
    k = n if form == 2 else 210
    A = rng.standard_normal((m, k))
    Bt = rng.standard_normal((n, k))
    if form == 2:
        Bt = np.tril(Bt) + np.tril(Bt, -1).T
    A[17] = 0.0
    A[17, 5] = value
    C0 = rng.standard_normal((m, n)) if form < 2 else np.zeros((m, n))
    got = product(ctx, form, 0, A, {0: Bt, 1: Bt.T, 2: np.tril(Bt)}[form], 1.0, 1.0 if form < 2 else 0.0, C0)
    want = A @ Bt.T + C0
    keep = np.arange(m) != 17
    assert np.allclose(got[keep], want[keep], rtol=1e-12, atol=1e-12)
    if form == 2 and np.isinf(value):
        # the FP64 path multiplies the operand's two masked triangles, whose zeros
        # turn an infinity into NaN in part of the row
        assert not np.isfinite(got[17]).any()
        return
    with np.errstate(invalid="ignore"):
        w17 = value * Bt[:, 5] + C0[17]
    assert np.array_equal(np.isnan(got[17]), np.isnan(w17))
    fin = np.isfinite(w17)
    assert np.array_equal(got[17][~fin & ~np.isnan(w17)], w17[~fin & ~np.isnan(w17)])
    assert np.allclose(got[17][fin], w17[fin], rtol=1e-12, atol=1e-12)


def test_wait_limit_does_not_reach_the_fp64_path(ctx):
    """A short wait limit of the mixed path's kernels leaves FP64 products alone."""
    rng = np.random.default_rng(2)
    A, B = values(rng, 300, 300), values(rng, 300, 300)
    ctx.set_wait_limit(1)
    try:
        got = product(ctx, 0, 0, A, B, 1.0, 0.0, np.zeros((300, 300)))
    finally:
        ctx.set_wait_limit(0)
    check_close(got, A, B, 1.0, 0.0, np.zeros((300, 300)))


def test_reconstructor_and_cee_at_a_size_that_uses_them(ctx):
    """nmeas 3,000 x nmeasts 2,500 with graded variables (diagonal from 1 to
    2^-40): R, L and Cee against torch's FP64, within 50 kappa eps of the
    equilibrated system."""
    import torch
    rng = np.random.default_rng(8)
    n, m, na = 3000, 2500, 700
    x = np.sort(rng.uniform(0, 60, n))
    S = np.exp(-np.abs(x[:, None] - x[None, :])) + 0.01 * np.eye(n)
    d = 2.0 ** np.linspace(0, -40, n).round()
    T = np.exp(-np.abs(rng.uniform(0, 60, m)[:, None] - x[None, :]))
    s, t, dd = gpu(S), gpu(T), gpu(d)
    w = torch.linalg.eigvalsh(s)
    tol = 50 * float(w[-1] / w[0]) * EPS
    Lw = torch.linalg.cholesky(s)
    Rw = torch.cholesky_solve(t.T, Lw)          # column-major R of the equilibrated system
    Cmm = torch.tril(dd[:, None] * s * dd[None, :]).T.contiguous()
    Ctm = (t * dd[None, :]).T.contiguous()
    keep = Cmm.clone()
    M.reconstructor(n, m, Cmm, n, Ctm, m, 1, ctx=ctx)
    R = Ctm * dd[:, None]                        # undo the grading
    assert float((R - Rw).norm() / Rw.norm()) <= tol
    L = torch.tril(Cmm.T) / dd[:, None]
    assert float((L - Lw).norm() / Lw.norm()) <= tol
    Ctt = torch.eye(m, dtype=torch.float64, device="cuda") * 2 + t @ t.T / n
    Dx = gpu(rng.standard_normal((m, na)))
    Cpm = (t * dd[None, :]).T.contiguous()
    Cpp = Ctt.clone()
    Cee, Cvv, Tmp = torch.zeros_like(Ctt), torch.zeros(na, na, dtype=torch.float64, device="cuda"), \
        torch.zeros(m, na, dtype=torch.float64, device="cuda")
    Rg = Ctm.clone()
    M.Cee_Cvv(n, m, na, keep, n, Cpp, m, Cpm, m, Rg, m, Dx, na, Cee, m, Cvv, na, Tmp, na, ctx=ctx)
    Rt = R.T
    CR = t @ Rt.T
    want = Ctt - CR - CR.T + Rt @ s @ Rt.T
    scale = float(CR.norm())
    assert float((Cee.T - want).norm()) <= 200 * math.sqrt(n) * EPS * scale
    wv = Dx.T @ want @ Dx
    assert float((Cvv.T - wv).norm() / wv.norm()) <= 200 * math.sqrt(n) * EPS * scale / float(want.norm())
