"""Calls captured into a CUDA graph: the covariance tiles, an FP64 Cee/Cvv large enough
for residue products, and a PSF. A first call may be the captured one, and a graph stays
valid whatever the context computes between its capture and its replay.

Covariances and the PSF have the same bits as in a plain call. Cee/Cvv runs on the FP64
tensor cores in the graph and by residues outside: each of its four chained products is
off by at most K eps |A| |B|, 8 K eps of the sum of the terms' absolute values between
the two."""
import os

import numpy as np
import pytest

import moao_b200 as M
from moao_b200 import inputs as I
from moao_b200 import params as P

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def r(g, *s):
    import torch
    return torch.randn(s, generator=g, device="cuda", dtype=torch.float64)


class Cee:
    def __init__(self, ctx, n, m, na, seed):
        import torch
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        self.ctx, self.size = ctx, (n, m, na)
        S = r(g, n, n)
        self.S, self.Ctt, self.Ctm, self.R, self.Dx = S @ S.T / n, r(g, m, m), r(g, n, m), r(g, n, m), r(g, m, na)
        self.Cpp, self.Cpm = self.Ctt.clone(), self.Ctm.clone()
        self.Cee, self.Cvv, self.Tmp = r(g, m, m), r(g, na, na), r(g, m, na)

    def run(self):
        n, m, na = self.size
        self.Cpp.copy_(self.Ctt)
        self.Cpm.copy_(self.Ctm)
        M.Cee_Cvv(n, m, na, self.S, n, self.Cpp, m, self.Cpm, m, self.R, m, self.Dx, na, self.Cee, m,
                  self.Cvv, na, self.Tmp, na, ctx=self.ctx)

    def bound(self):
        import torch
        n = self.size[0]
        aR, aC = self.R.T.abs(), self.Ctm.T.abs()
        t = self.Ctt.abs() + aC @ aR.T + aR @ aC.T + aR @ (self.S.abs() @ aR.T)
        return 8 * n * EPS * torch.maximum(t, t.T)


def on_stream(f):
    """f(ctx, stream) on a context of its own that runs on a side stream."""
    import torch
    st = torch.cuda.Stream()
    ctx = M.Context(0)
    ctx.set_stream(st.cuda_stream)
    try:
        with torch.cuda.stream(st):
            f(ctx, st)
            torch.cuda.synchronize()
    finally:
        ctx.close()


@pytest.mark.parametrize("warm", [False, True])
def test_cee(built, cuda, warm):
    import torch

    def body(ctx, st):
        c = Cee(ctx, 3000, 1500, 400, 1)
        big = Cee(ctx, 3500, 2000, 500, 2)
        if warm:
            c.run()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            c.run()
        big.run()  # grows the context's buffers
        c.Cee.zero_()
        g.replay()
        torch.cuda.synchronize()
        got = c.Cee.clone()
        c.run()
        torch.cuda.synchronize()
        assert bool(((got - c.Cee).abs() <= c.bound()).all())

    on_stream(body)


def test_covariance_and_psf(built, cuda, tmp_path):
    import torch
    s, a = P.config_scaled(12, 5, 1, 3, 2)
    P.write_system(str(tmp_path), s, a)
    t = M.Tomo(os.path.join(tmp_path, "sys-params.txt"), os.path.join(tmp_path, "prof-1-atmos-night0.txt"))
    t.setTarget(0)
    nm, nts = t.getNMeas(), t.getNMeasTS()
    ins = I.intersample_inputs(12, 39.0, 0.28)

    def body(ctx, st):
        z = lambda *x: torch.zeros(x, dtype=torch.float64, device="cuda")  # noqa: E731
        C, T, S, p = z(nm, nm), z(nm, nts), z(nts, nts), z(512, 512)
        isx = M.Intersample(ins.nact ** 2, ins.np_, 39.0, ins.idx, ins.abs2fi, ins.otf, ctx=ctx)
        cvv = torch.from_numpy(np.random.default_rng(1).random((ins.nact, ins.nact)) * 1e-3).cuda()
        M.matcov_tile(S, 1, 1, 0, 0, nts, t, 4, ctx=ctx)  # the geometry, uploaded outside the graph

        def run():
            M.matcov_tile(C, nm, nm, 0, 0, nm, t, 1, ctx=ctx)
            M.matcov_tile(T, nts, nm, 0, 0, nts, t, 3, ctx=ctx)
            M.matcov_tile(S, nts, nts, 0, 0, nts, t, 4, ctx=ctx)
            isx.process(cvv, out=p)

        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            run()
        g.replay()
        torch.cuda.synchronize()
        got = [x.clone() for x in (C, T, S, p)]
        for x in (C, T, S, p):
            x.zero_()
        run()
        torch.cuda.synchronize()
        for x, y in zip(got, (C, T, S, p)):
            assert torch.equal(x, y) and bool((x != 0).any())
        isx.close()

    on_stream(body)
