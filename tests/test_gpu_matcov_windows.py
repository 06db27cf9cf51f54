"""Windows of a large system's covariance matrices: only the cell tiles that hold their
subapertures are visited. The elements have the bits of a larger window's (whatever the
tiles' rows it begins and ends in), and a window's time does not grow with the system:
at most twice that of the same window in a system of a sixteenth of the subapertures
(visiting all tile pairs it was 3 to 6 times)."""
import os

import numpy as np
import pytest

import moao_b200 as M
from moao_b200 import params as P

pytestmark = pytest.mark.gpu


def tomo(tmp_path, nssp):
    s, a = P.config_scaled(nssp, 2, 1, 3, 2)
    d = os.path.join(tmp_path, str(nssp))
    P.write_system(d, s, a)
    t = M.Tomo(os.path.join(d, "sys-params.txt"), os.path.join(d, "prof-1-atmos-night0.txt"))
    t.setTarget(0)
    return t


def tile(ctx, t, typ, nr, nc, x0, y0):
    import torch
    d = torch.full((nc, nr), 7.0, dtype=torch.float64, device="cuda")
    M.matcov_tile(d, nr, nc, x0, y0, nr, t, typ, ctx=ctx)
    ctx.synchronize()
    return d.T


@pytest.mark.parametrize("nssp", [17, 32])
def test_bits(tmp_path, ctx, nssp):
    """Every slope of one LGS against windows that begin and end anywhere in an NGS."""
    import torch
    t = tomo(tmp_path, nssp)
    nm, nts = t.getNMeas(), t.getNMeasTS()
    whole = {1: tile(ctx, t, 1, nm, nm, 0, 0), 2: tile(ctx, t, 2, nm, nts, 0, 0),
             3: tile(ctx, t, 3, nts, nm, 0, 0)}
    rng = np.random.default_rng(nssp)
    for typ, m in whole.items():
        h, w = m.shape
        for k in range(40):
            nr, nc = (1, w) if k % 2 else (h, 1)
            if k >= 20:
                nr, nc = int(rng.integers(1, h // 4)), int(rng.integers(1, w // 4))
            x0, y0 = int(rng.integers(0, h - nr + 1)), int(rng.integers(0, w - nc + 1))
            assert torch.equal(tile(ctx, t, typ, nr, nc, x0, y0), m[x0:x0 + nr, y0:y0 + nc]), (typ, nr, nc, x0, y0)


def test_time_does_not_grow_with_the_system(tmp_path, ctx):
    import torch
    buf = torch.empty(64 * 64, dtype=torch.float64, device="cuda")
    s = torch.cuda.ExternalStream(ctx.stream)
    ms = {}
    for nssp in (16, 64):
        t = tomo(tmp_path, nssp)
        nm = t.getNMeas()
        for h, w in ((64, 64), (1, 1)):
            best = 1e9
            for _ in range(20):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(s)
                M.matcov_tile(buf, h, w, nm - h - 5, 5, h, t, 1, ctx=ctx)
                b.record(s)
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            ms[nssp, h] = best
    assert ms[64, 64] <= 2 * ms[16, 64] and ms[64, 1] <= 2 * ms[16, 1], ms
