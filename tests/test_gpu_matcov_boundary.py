"""Separations of exactly 0.75 L0, where the model's structure function passes from its
series to its asymptotic form with a jump of 5e-7: a subaperture grid whose pitch divides
0.75 L0 holds them, and the series applies to them (x > Xlim is false). Covariances of
the LGS/NGS pairs, the equal-projection pairs and Ctt against the oracle, to 1e-11 of the
matrix maximum (the bound of test_gpu_matcov_edge.py; a separation on the wrong side is
off by 1e-7)."""
import os

import numpy as np
import pytest

import moao_b200 as M
import oracle as O
from moao_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nssp,pitch,L0", [(6, 0.5, 2.0), (13, 0.5, 4.0), (20, 0.5, 8.0), (10, 0.75, 4.0),
                                           (16, 1.0, 16.0), (9, 0.25, 1.0)])
def test_series_at_the_boundary(tmp_path, ctx, nssp, pitch, L0):
    import torch
    s = P.make_sys(pitch * nssp, 0.14, nssp, 2, 2, 30.0, np.random.default_rng(nssp))
    a = P.make_atm([0.0, 3000.0], [0.6, 0.4], 0.13, [L0, 25.0])
    P.write_system(str(tmp_path), s, a)
    t = M.Tomo(os.path.join(tmp_path, "sys-params.txt"), os.path.join(tmp_path, "prof-1-atmos-night0.txt"))
    t.setTarget(0)
    g = O.Geometry.from_tomo(t)
    for typ, h, w in ((1, g.nmeas, g.nmeas), (3, g.nmeasts, g.nmeas), (4, g.nmeasts, g.nmeasts)):
        want = O.matcov(g, h, w, 0, 0, typ)
        d = torch.zeros((w, h), dtype=torch.float64, device="cuda")
        M.matcov_tile(d, h, w, 0, 0, h, t, typ, ctx=ctx)
        ctx.synchronize()
        got = d.T.cpu().numpy().copy()
        if typ == 1:
            want, got = np.tril(want), np.tril(got)
        err = np.abs(got - want).max() / np.abs(want).max()
        assert err <= 1e-11, (typ, err)
