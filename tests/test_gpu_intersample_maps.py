"""The covariance-map step of the intersample PSF on both of its routes: partial
maps by columns of Cvv (a square Cvv, every column's entries in different cells)
and a warp per cell (any other index table), at the sizes where they can go wrong:
one actuator, fewer columns than CTAs, a column of more than 4,096 entries, a map
too large for shared memory, cells never or often hit.

Oracle: the numpy restatement of the pipeline. Tolerance 1e-10 of the PSF's peak,
as in the other PSF tests: a cell's sum of n entries is off by at most n eps of
their magnitudes (n up to 10,000 here, 2e-12), and the exponent of the structure
function, of order one at these amplitudes, carries that over."""
import numpy as np
import pytest

import oracle as O
import moao_b200 as M
from moao_b200 import inputs as I

pytestmark = pytest.mark.gpu


def cvv_of(n, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((n, 8)) * 0.05
    return B @ B.T + 0.01 * np.eye(n)


def run(ctx, nssp, idx, C):
    x = I.intersample_inputs(nssp, 39.0, 0.28)
    want = O.intersample(C, idx, x.abs2fi, x.otf, x.np_)
    isx = M.Intersample(idx.size, x.np_, 39.0, idx, x.abs2fi, x.otf, ctx=ctx)
    got = isx.process(np.asfortranarray(C))
    again = isx.process(np.asfortranarray(C))
    isx.close()
    assert np.array_equal(got, again)
    assert np.max(np.abs(got - want)) <= 1e-10 * np.max(np.abs(want))


def spread(n, nmap):
    """1-based cells, different within a column of n entries."""
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    return ((11 * i + 13 * j) % nmap + 1).astype(np.int64).flatten("F")


@pytest.mark.parametrize("nssp,n", [(10, 1), (10, 7), (10, 100), (24, 600), (79, 4100)])
def test_columns(ctx, nssp, n):
    nmap = (2 * nssp + 1) ** 2
    assert np.gcd(11, nmap) == 1 and n <= nmap
    run(ctx, nssp, spread(n, nmap), cvv_of(n, n))


@pytest.mark.parametrize("nssp,n", [(10, 7), (10, 100), (24, 300)])
def test_repeated_cells_in_a_column(ctx, nssp, n):
    rng = np.random.default_rng(n)
    idx = rng.integers(1, (2 * nssp + 1) ** 2 + 1, n * n)
    idx[: n * n // 2] = 5  # one cell takes half of the entries
    run(ctx, nssp, idx, cvv_of(n, n))


def test_map_beyond_shared_memory(ctx):
    nssp, n = 84, 500  # 169^2 cells: 228 KB
    run(ctx, nssp, spread(n, (2 * nssp + 1) ** 2), cvv_of(n, 3))


def test_table_that_is_not_square(ctx):
    x = I.intersample_inputs(10, 39.0, 0.28)
    rng = np.random.default_rng(4)
    idx = rng.integers(1, 21 ** 2 + 1, 50 * 51)
    C = cvv_of(51, 9)[:, :50]
    want = O.intersample(C, idx, x.abs2fi, x.otf, x.np_)
    isx = M.Intersample(idx.size, x.np_, 39.0, idx, x.abs2fi, x.otf, ctx=ctx)
    got = isx.process(np.asfortranarray(C).flatten("F"))
    isx.close()
    assert np.max(np.abs(got - want)) <= 1e-10 * np.max(np.abs(want))
