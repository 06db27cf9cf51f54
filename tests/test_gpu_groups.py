"""The FP64 reconstructor at sizes whose panels are taken in groups (residue products):
whole groups, a last group of one panel, panels of 1, 64 and 960 columns at the end, and a
size with one group only; a pivot that fails in a group's second panel.

Oracle: torch's FP64 factor and solves. Tolerance: two correct FP64 solves agree to
O(kappa eps), 50 of it as elsewhere, kappa of the equilibrated system."""
import numpy as np
import pytest

import moao_b200 as M

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def system(n, m):
    import torch
    rng = np.random.default_rng(n)
    x = torch.from_numpy(np.sort(rng.uniform(0, 60, n))).cuda()
    y = torch.from_numpy(rng.uniform(0, 60, m)).cuda()
    s = torch.exp(-(x[:, None] - x[None, :]).abs()) + 0.01 * torch.eye(n, dtype=x.dtype, device="cuda")
    d = 2.0 ** torch.linspace(0, -40, n, dtype=x.dtype, device="cuda").round()
    t = torch.exp(-(y[:, None] - x[None, :]).abs())
    return s, d, t


@pytest.mark.parametrize("n", [4096, 5 * 1024 + 1, 6 * 1024, 7 * 1024 + 64, 8 * 1024 - 64])
def test_reconstructor_in_groups(ctx, n):
    import torch
    m = 2200
    s, d, t = system(n, m)
    w = torch.linalg.eigvalsh(s)
    tol = 50 * float(w[-1] / w[0]) * EPS
    Lw = torch.linalg.cholesky(s)
    Rw = torch.cholesky_solve(t.T, Lw)
    Cmm = torch.tril(d[:, None] * s * d[None, :]).T.contiguous()
    Ctm = (t * d[None, :]).T.contiguous()
    M.reconstructor(n, m, Cmm, n, Ctm, m, 1, ctx=ctx)
    R = Ctm * d[:, None]
    assert float((R - Rw).norm() / Rw.norm()) <= tol
    L = torch.tril(Cmm.T) / d[:, None]
    assert float((L - Lw).norm() / Lw.norm()) <= tol


def test_failing_pivot_in_a_group(ctx):
    n, m, bad = 6 * 1024, 64, 3 * 1024 + 777
    s, d, t = system(n, m)
    s[bad, bad] = -1.0
    Cmm, Ctm = s.T.contiguous(), t.T.contiguous()
    with pytest.raises(M.NotSPDError) as e:
        M.reconstructor(n, m, Cmm, n, Ctm, m, 1, ctx=ctx)
    assert str(bad + 1) in str(e.value)
