"""The buffers of the FP64 residue products are kept on a context between calls, but no
call fails for want of the memory they hold: an allocation that does not fit beside them
takes their room. A full device is stood in for by the context's limit on held bytes;
for the batch engine, which asks the device, by filling it."""
import os

import numpy as np
import pytest

import moao_b200 as M
from moao_b200 import batch as B
from moao_b200 import params as P
from moao_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def held(ctx):
    return lib().moao_debug_bytes_held(ctx.handle)


def limit(ctx, nbytes):
    check(lib().moao_debug_limits(ctx.handle, nbytes, 0, 0), "limits")


def system(n, m, seed=1):
    """A well-conditioned Cmm, a Ctm and their reconstructor."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.rand(n, generator=g, dtype=torch.float64, device="cuda") * n ** 0.5
    C = torch.exp(-(x[:, None] - x[None, :]).abs()) + torch.eye(n, dtype=torch.float64, device="cuda")
    T = torch.randn((n, m), generator=g, dtype=torch.float64, device="cuda")
    return C, T, torch.cholesky_solve(T, torch.linalg.cholesky(C))


def rec(ctx, n, m, C, T, prec="fp64"):
    c, t = C.clone(), T.clone()
    M.reconstructor(n, m, c, n, t, m, 1, prec=prec, ctx=ctx)
    ctx.synchronize()
    return t


def rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.fixture
def own(built, cuda):
    c = M.Context(0)
    yield c
    c.close()


def fill(ctx):
    """An FP64 reconstructor whose products go by residues; what it needs without."""
    n, m = 4096, 1500
    C, T, R = system(n, m)
    assert rel(rec(ctx, n, m, C, T), R) <= 1e-10   # kappa is below 2 sqrt(n): 1e4 eps covers it
    need = 8 * 1024 * 2 * n                        # panels and inverse blocks
    assert held(ctx) > 2 * need
    return need


def test_mixed_after_fp64(own, built):
    need = fill(own)
    n, m = 3000, 400
    C, T, R = system(n, m, 2)
    probe = M.Context(0)
    rec(probe, n, m, C, T, "mixed")
    mixed = held(probe)
    probe.close()
    limit(own, need + mixed + 1_000_000)
    assert held(own) + mixed > need + mixed + 1_000_000
    assert rel(rec(own, n, m, C, T, "mixed"), R) <= 1e-5
    assert held(own) <= need + mixed + 1_000_000


def test_larger_fp64_runs_without_residues(own):
    """Room for the panels of a larger system, not for its residues."""
    fill(own)
    n, m = 6000, 1500
    C, T, R = system(n, m, 3)
    cap = 8 * 1024 * 2 * n + 8_000_000
    limit(own, cap)
    assert rel(rec(own, n, m, C, T), R) <= 1e-10
    assert held(own) <= cap


def test_host_paths_after_fp64(own):
    need = fill(own)
    n, m, na = 300, 200, 100
    rng = np.random.default_rng(5)
    host = [rng.standard_normal(s) for s in ((n, n), (m, m), (n, m), (n, m), (m, na), (m, m), (na, na), (m, na))]
    limit(own, need + 3_000_000)
    lds = [n, m, m, m, na, m, na, na]
    args = [x for p in zip(host, lds) for x in p]
    M.Cee_Cvv(n, m, na, *args, ctx=own)
    assert held(own) <= need + 3_000_000


def test_batch_after_fp64(own, tmp_path):
    """The device filled so that one instance fits only with the residues' room."""
    import torch
    tomos = []
    for k, nssp in enumerate((8, 24)):
        s, a = P.config_scaled(nssp, 2)
        d = os.path.join(tmp_path, str(k))
        P.write_system(d, s, a)
        tomos.append(M.Tomo(os.path.join(d, "sys-params.txt"), os.path.join(d, "prof-1-atmos-night0.txt")))
    outs = [torch.zeros(t.getNMeas() * t.getNMeasTS(), dtype=torch.float64, device="cuda") for t in tomos]
    n, m = tomos[1].getNMeas(), tomos[1].getNMeasTS()
    need = 8 * (n * n + m * n + 1024 * 2 * n)

    def batch(k):
        per, _ = B.batch_reconstructors([tomos[k]], [outs[k]], packed_max=-1, ctx=own)
        return per[0]["status"]

    assert batch(0) == 0          # modules loaded, the sub-context made
    C, T, _ = system(8192, 2500)
    rec(own, 8192, 2500, C, T)
    del C, T
    residues = held(own) - 8 * 1024 * 2 * 8192
    assert residues > need
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill_up = torch.empty(free - int(0.9 * need), dtype=torch.uint8, device="cuda")
    try:
        assert batch(1) == 0
    finally:
        del fill_up
        torch.cuda.empty_cache()
    got = outs[1].clone()
    assert batch(1) == 0
    assert torch.equal(got, outs[1]) and bool(torch.isfinite(got).all())


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_server_stays_in_its_budget(built, cuda, tmp_path, prec):
    """A budget without room for residue buffers: the request runs, its result is that of
    a roomy server within the FP64 products' accuracy (kappa of these systems is below
    1e6, so 1e-9 covers n eps kappa), and the slot's memory stays inside the budget."""
    import torch
    from moao_b200.serve import Server
    s, a = P.config_scaled(24, 3)
    P.write_system(str(tmp_path), s, a)
    files = os.path.join(tmp_path, "sys-params.txt"), os.path.join(tmp_path, "prof-1-atmos-night0.txt")
    prof = np.array(a.cn2), np.array(a.h), np.array(a.L0)
    out, foot = [], None
    for k in range(2):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        budget = 60.0 if k == 0 else 1.001 * foot
        with Server(slots=1, hbm_budget_gb=budget) as srv:
            sid = srv.add_system(*files)
            info = srv.system_info(sid)
            R = np.zeros(info["nmeas"] * info["nmeasts"])
            r = srv.wait(srv.submit(sid, *prof, prec=prec, R=R))
            assert r["status"] == 0, r
            foot = r["footprint_gb"]
            used = (free - torch.cuda.mem_get_info()[0]) / 1e9
            admitted = srv.stats()["peak_admitted_gb"]
            # streams, modules and the structure-function table come on top
            assert used <= admitted + 0.1, (used, admitted, foot)
            assert admitted <= budget
            if prec == "fp64":
                assert (admitted > 1.2 * foot) == (k == 0)
        out.append(R)
    assert np.linalg.norm(out[0] - out[1]) <= 1e-9 * np.linalg.norm(out[1])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_a_destroyed_context_leaves_nothing(built, cuda, prec):
    import torch
    n, m = 4000, 800
    C, T, _ = system(n, m)
    free = []
    for _ in range(3):
        ctx = M.Context(0)
        rec(ctx, n, m, C, T, prec)
        torch.cuda.synchronize()
        kept = held(ctx)
        before = torch.cuda.mem_get_info()[0]
        ctx.close()
        free.append(torch.cuda.mem_get_info()[0])
        # everything counted as held comes back (cudaMalloc rounds each buffer up to 2 MB)
        assert free[-1] - before >= 0.95 * kept
    assert free[0] - free[-1] <= 32e6, free
