"""Covariances whose WFS pairs meet at cell edges (LGS against NGS, truth sensor
against LGS), and Ctt, where the grid leaves remainders of the 4x4 and 8x8 cell
tiles, over layers whose outer scales put separations below, inside and above the
tabulated range of the structure function (exact zeros included), one of them above
the guide star (masked).

Tolerance: 1e-11 of the matrix maximum, against the oracle. Each value of f carries a
few units of 2^-53 on both sides, with a separation of up to 10^2 subapertures against
the diagonal's one: (10^2)^(5/3) = 2000 times 4 * 2^-53 over 7 layers is 6e-12.
"""
import os

import numpy as np
import pytest

import moao_b200 as M
import oracle as O
from moao_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nssp", [3, 4, 5, 7, 8, 9, 13, 17])
def test_edge_pairs_and_ctt(tmp_path, ctx, nssp):
    import torch
    rng = np.random.default_rng(nssp)
    s = P.make_sys(0.5 * nssp, 0.14, nssp, 2, 2, 30.0, rng)
    a = P.make_atm([0.0, 0.0, 500.0, 4000.0, 9000.0, 20000.0, 120000.0],
                   [0.3, 0.2, 0.1, 0.1, 0.1, 0.1, 0.1], 0.13, [25.0, 1e5, 0.05, 0.7, 6.0, 400.0, 20.0])
    P.write_system(str(tmp_path), s, a)
    t = M.Tomo(os.path.join(tmp_path, "sys-params.txt"), os.path.join(tmp_path, "prof-1-atmos-night0.txt"))
    g = O.Geometry.from_tomo(t)
    nm, nts = g.nmeas, g.nmeasts
    ctm = O.matcov(g, nts, nm, 0, 0, 3)
    cmm = O.matcov(g, nm, nm, 0, 0, 1)
    want = {1: cmm, 5: np.tril(cmm) + np.tril(cmm, -1).T, 3: ctm, 2: ctm.T,
            4: O.matcov(g, nts, nts, 0, 0, 4)}
    for typ, ref in want.items():
        h, w = ref.shape
        for x0, y0 in ((0, 0), (h // 3, h // 3 if typ == 5 else w // 5)):  # the whole matrix; a ragged window of it
            nr, nc = h - x0, w - y0
            d = torch.full((nc, nr + 3), 7.0, dtype=torch.float64, device="cuda")
            M.matcov_tile(d, nr, nc, x0, y0, nr + 3, t, typ, ctx=ctx)
            ctx.synchronize()
            got = d.cpu().numpy().T
            assert np.all(got[nr:] == 7.0)
            part = ref[x0:, y0:].copy()
            if typ == 1:
                upper = np.arange(nr)[:, None] + x0 < np.arange(nc)[None, :] + y0
                assert np.all(got[:nr][upper] == 7.0)
                part[upper] = 7.0
            assert np.all(np.isfinite(part))
            err = np.abs(got[:nr] - part).max() / np.abs(ref).max()
            assert err <= 1e-11, (typ, x0, y0, err)
