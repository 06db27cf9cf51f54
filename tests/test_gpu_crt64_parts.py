"""FP64 residue products taken in parts (operands' rows that do not fit the residue
buffers at once, more tiles than one launch takes) and where the buffers do not fit
the device.

The residues, their sums and each element's reconstruction do not depend on the parts,
so the results have the same bits as in one part. Where the guard sends a part to the
FP64 tensor cores, the bound is that of test_gpu_crt64.py (which covers both kernels).
A call that finds no room for its buffers is an FP64 call like any other: each of its
products is off by at most K eps |A| |B|; four of them in a chain, on a residue run and
an FP64 run, stay within 8 K eps of the sum of the terms' absolute values."""
import numpy as np
import pytest

import moao_b200 as M
from moao_b200._lib import check, lib
from test_gpu_crt64 import EPS, check_close, product, values

pytestmark = pytest.mark.gpu


@pytest.fixture
def own(built, cuda):
    c = M.Context(0)
    yield c
    c.close()


def limits(ctx, workspace=0, operand=0, tiles=0):
    check(lib().moao_debug_limits(ctx.handle, workspace, operand, tiles), "limits")


def in_parts(ctx, *args):
    """256 rows of an operand and two tiles at a time."""
    limits(ctx, operand=1, tiles=2)
    try:
        return product(ctx, *args)
    finally:
        limits(ctx)


@pytest.mark.parametrize("form,m,n,k", [(0, 700, 900, 300), (0, 257, 513, 1100), (1, 600, 300, 129),
                                        (1, 256, 770, 1), (2, 600, 1111, 1111), (2, 3, 513, 513)])
def test_parts_give_the_same_bits(own, form, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A, B = values(rng, m, k), values(rng, n, k)
    if form == 1:
        B = B.T
    elif form == 2:
        B = np.tril(B) + np.triu(np.full((k, k), np.nan), 1)
    C0 = rng.standard_normal((m, n))
    args = (form, 0, A, B, 1.0 if form == 2 else -0.5, 0.0 if form == 2 else 1.0, C0)
    assert np.array_equal(in_parts(own, *args), product(own, *args))


@pytest.mark.parametrize("n,k", [(300, 40), (700, 300), (1025, 130)])
def test_lower_parts_give_the_same_bits(own, n, k):
    rng = np.random.default_rng(n)
    A, B = values(rng, n, k), values(rng, n, k)
    C0 = rng.standard_normal((n, n))
    for other in (A, B):
        args = (0, 1, A, other, -1.0, 1.0, C0)
        got = in_parts(own, *args)
        assert np.array_equal(got, product(own, *args))
        up = np.triu(np.ones((n, n), bool), 1)
        assert np.array_equal(got[up], C0[up])


@pytest.mark.parametrize("form,lower", [(0, 0), (0, 1), (1, 0), (2, 0)])
@pytest.mark.parametrize("row", [20, 300])
def test_guard_in_one_part(own, form, lower, row):
    """A NaN in one part of the rows: that part by the FP64 tensor cores, tile range by
    tile range, the others by residues."""
    rng = np.random.default_rng(row)
    m = n = 650
    k = 650 if form == 2 else 210
    A, Bt = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    if form == 2:
        Bt = np.tril(Bt) + np.tril(Bt, -1).T
    beta = 0.0 if form == 2 else 1.0
    C0 = rng.standard_normal((m, n)) * beta
    keep = np.ones((m, n), bool)
    keep[row] = False
    if lower:
        keep &= np.tril(np.ones((m, n), bool))
    clean = A.copy()
    clean[row] = 0.0
    A[row, 5] = np.nan
    got = in_parts(own, form, lower, A, {0: Bt, 1: Bt.T, 2: np.tril(Bt)}[form], 1.0, beta, C0)
    check_close(got, clean, Bt, 1.0, beta, C0, keep, sym=form == 2)
    last = row + 1 if lower else n
    assert np.isnan(got[row, :last]).all()
    assert np.array_equal(got[row, last:], C0[row, last:])


def test_no_room_for_a_later_part(built, cuda):
    """Cee of nmeasts 3,000 with operands in parts of 1,536 rows: the first part of a
    lower product is a triangle of 42 tiles, the second a square of 72. Room for the
    first only: the products run on the FP64 tensor cores, and nothing is added twice."""
    import torch
    n, m, na = 1100, 3000, 300
    g = torch.Generator(device="cuda")
    g.manual_seed(4)

    def r(*s):
        return torch.randn(s, generator=g, device="cuda", dtype=torch.float64)

    S = r(n, n)
    S = S @ S.T / n
    Ctt, Ctm, R, Dx = r(m, m), r(n, m), r(n, m), r(m, na)
    row = 16 * 1152
    outs = []
    for cap in (0, 2 * 1536 * row + 30_000_000):
        ctx = M.Context(0)
        limits(ctx, workspace=cap, operand=1536 * row)
        Cpp, Cpm = Ctt.clone(), Ctm.clone()
        Cee, Cvv, Tmp = torch.zeros_like(Ctt), r(na, na), r(m, na)
        M.Cee_Cvv(n, m, na, S, n, Cpp, m, Cpm, m, R, m, Dx, na, Cee, m, Cvv, na, Tmp, na, ctx=ctx)
        ctx.synchronize()
        held = lib().moao_debug_bytes_held(ctx.handle)
        assert held <= cap if cap else held > 2 * 1536 * row + 30_000_000
        outs.append((Cee, Cvv))
        ctx.close()
    aR, aS, aC = R.T.abs(), S.abs(), Ctm.T.abs()
    terms = Ctt.abs() + aC @ aR.T + aR @ aC.T + aR @ (aS @ aR.T)
    lim = 8 * n * EPS * terms
    # only Ctt's lower triangle counts, in both halves of Cee
    lim = torch.maximum(lim, lim.T)
    assert bool(((outs[0][0] - outs[1][0]).abs() <= lim).all())
    D = Dx.T.abs()
    lim = D @ lim @ D.T + 8 * m * EPS * (D @ torch.maximum(terms, terms.T) @ D.T)
    assert bool(((outs[0][1] - outs[1][1]).abs() <= lim).all())
