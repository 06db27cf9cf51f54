"""The work that a user of this library has it do, as cases to be timed.

A case is a dict of plain values; ``prepare`` makes its inputs from a seed,
``run`` takes them once through the public entry points and returns every
output, ``exact`` computes the same outputs in plain torch / numpy in 64 bits,
and ``work`` counts the bytes and operations that the case cannot do without.

Kinds of work (the stages of a tomographic-reconstructor refresh):

``cov``    a new turbulence profile, then the covariance matrices Cmm (lower),
           Ctm and Ctt generated from it: what starts every refresh.
``rec``    R = Ctm Cmm^-1 in FP64 or on the mixed-precision path, for one or
           several targets. Cmm is kept (the error budget needs it again), so a
           pass copies it into the buffer that the factor overwrites.
``cee``    the error covariance Cee and its actuator projection Cvv, FP64 or
           mixed.
``psf``    the long-exposure PSF of a Cvv.
``batch``  many small uneven systems built in one call (a survey of guide-star
           configurations).

Systems are those of ``moao_b200.params``: the 8 m system, the 39 m system at a
number of subapertures across, and random small ones. ``rec`` and ``cee`` take
covariances of the same systems' geometry under a Matern-5/2 phase model
computed here in torch (closed-form slope covariances, so the matrices are
positive definite and independent of the library's own covariance kernels),
with the WFS noise and LGS constants at the magnitudes of the real ones.
"""
import math
import os
import tempfile

import numpy as np
import torch

import moao_b200 as M
from moao_b200 import batch as B
from moao_b200 import inputs as I
from moao_b200 import params as P

DEV = "cuda"
F64 = torch.float64
RASC = 206265.0

_CTX = None


def _context():
    """One library context per process, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = M.Context(torch.cuda.current_device())
    return _CTX


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the 8 m system of the tests (nmeas 640): launches and latency count
        {"name": "cov_8m", "kind": "cov", "system": "8m", "nssp": 10, "nlgs": 3, "nngs": 1, "nlayer": 3},
        # an ordinary 39 m system on a 29 grid with 10 layers (nmeas ~ 8,000)
        {"name": "cov_29", "kind": "cov", "system": "39m", "nssp": 29, "nlgs": 4, "nngs": 3, "nlayer": 10},
        # the ELT system of the benchmark: 64 x 64, 35 layers (nmeas 47,552)
        {"name": "cov_elt", "kind": "cov", "system": "39m", "nssp": 64, "nlgs": 6, "nngs": 2, "nlayer": 35},
        # the 8 m reconstructor (nmeas 640): the refresh of a small instrument
        {"name": "rec_8m_fp64", "kind": "rec", "system": "8m", "nssp": 10, "nlgs": 3, "nngs": 1,
         "prec": "fp64", "ngal": 1},
        # a mid-size system, two targets from one factorisation (nmeas ~ 6,600)
        {"name": "rec_24_fp64", "kind": "rec", "system": "39m", "nssp": 24, "nlgs": 6, "nngs": 2,
         "prec": "fp64", "ngal": 2},
        # the largest system of the uneven batch (nmeas ~ 29,000) in FP64
        {"name": "rec_50_fp64", "kind": "rec", "system": "39m", "nssp": 50, "nlgs": 6, "nngs": 2,
         "prec": "fp64", "ngal": 1},
        # a mid-size system on the mixed path (nmeas ~ 12,000)
        {"name": "rec_32_mixed", "kind": "rec", "system": "39m", "nssp": 32, "nlgs": 6, "nngs": 2,
         "prec": "mixed", "ngal": 1},
        # the benchmark's own solve: the ELT system on the mixed path
        {"name": "rec_elt_mixed", "kind": "rec", "system": "39m", "nssp": 64, "nlgs": 6, "nngs": 2,
         "prec": "mixed", "ngal": 1},
        # error budget of a large system in FP64 (nmeas ~ 29,000)
        {"name": "cee_50_fp64", "kind": "cee", "system": "39m", "nssp": 50, "nlgs": 6, "nngs": 2,
         "prec": "fp64"},
        # error budget of a mid-size system on the mixed path (nmeas ~ 12,000)
        {"name": "cee_32_mixed", "kind": "cee", "system": "39m", "nssp": 32, "nlgs": 6, "nngs": 2,
         "prec": "mixed"},
        # the ELT system's PSF (512 x 512)
        {"name": "psf_64", "kind": "psf", "nssp": 64},
        # 24 uneven small systems in one launch
        {"name": "batch_24", "kind": "batch", "count": 24, "lo": 8, "hi": 20, "prec": "fp64",
         "packed": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng):
    kind = rng.choice(["cov", "cov", "rec", "rec", "rec", "cee", "cee", "psf", "batch"])
    if kind == "psf":
        return {"kind": kind, "nssp": _log_int(rng, 8, 64)}
    if kind == "batch":
        lo = rng.randint(6, 12)
        return {"kind": kind, "count": rng.randint(4, 24), "lo": lo, "hi": lo + rng.randint(2, 10),
                "prec": "fp64", "packed": rng.choice([-1, 2048, 4096])}
    c = {"kind": kind, "system": "39m", "nlgs": rng.randint(1, 6), "nngs": rng.randint(1, 3)}
    if kind == "cov":
        c.update(nssp=_log_int(rng, 8, 60), nlayer=rng.randint(1, 35))
    elif kind == "rec":
        c.update(prec=rng.choice(["fp64", "mixed"]), ngal=rng.randint(1, 2))
        c.update(nssp=_log_int(rng, 8, 50 if c["prec"] == "fp64" else 56))
        if c["nssp"] > 40:
            c["ngal"] = 1
    else:
        c.update(prec=rng.choice(["fp64", "mixed"]), nssp=_log_int(rng, 8, 50))
    return c


# ---------------------------------------------------------- systems, geometry
def _system(case, seed):
    nl = case.get("nlayer", 3)
    if case["system"] == "8m":
        s, a = P.config_small(seed)
    else:
        s, a = P.config_scaled(case["nssp"], nl, seed, case["nlgs"], case["nngs"])
    return s, a


def _survey(case, seed):
    """Uneven small systems: their sizes from the case, the turbulence profile
    (layers, strengths, outer scales) from the seed."""
    sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    rng = np.random.default_rng(int(seed))
    out = []
    for _ in range(case["count"]):
        s, a = P.config_random(sizes, nssp_range=(case["lo"], case["hi"]), nwfs_range=(2, 5),
                               nlayer_range=(1, 8))
        nl = a.nLayer
        out.append((s, P.make_atm(np.sort(rng.uniform(0.0, 20000.0, nl)), rng.dirichlet(np.ones(nl)),
                                  float(rng.uniform(0.08, 0.2)), rng.uniform(10.0, 50.0, nl))))
    return out


def _centres(s):
    """Valid subaperture centres of one WFS (row-major over the grid)."""
    pas = s.diam / s.nssp
    c = -s.diam / 2.0 + pas / 2.0 * (2.0 * torch.arange(s.nssp, dtype=F64) + 1.0)
    y, x = torch.meshgrid(c, c, indexing="ij")
    r2 = x * x + y * y
    robs = 0.285 if s.nssp == 7 and 0.285 < s.obs < 0.29 else s.obs
    ok = ~((r2 < (s.diam * robs / 2.0) ** 2) | (r2 >= s.diam * s.diam / 4.0))
    return x[ok].to(DEV), y[ok].to(DEV)


def _sizes(case):
    s, _ = _system(case, 1)
    n = _centres_count(s)
    return 2 * n * (s.nW - 1), 2 * n


def _centres_count(s):
    pas = s.diam / s.nssp
    c = -s.diam / 2.0 + pas / 2.0 * (2.0 * np.arange(s.nssp) + 1.0)
    r2 = c[:, None] ** 2 + c[None, :] ** 2
    robs = 0.285 if s.nssp == 7 and 0.285 < s.obs < 0.29 else s.obs
    return int((~((r2 < (s.diam * robs / 2.0) ** 2) | (r2 >= s.diam ** 2 / 4.0))).sum())


def _projected(s, w, h, x, y):
    """Subaperture centres of WFS w on the layer at altitude h (no rotation)."""
    rr = 1.0 - h * s.gsAlt[w]
    return ((x + s.XPup[w]) * rr + s.alphaX_as[w] / RASC * h,
            (y + s.YPup[w]) * rr + s.alphaY_as[w] / RASC * h)


def _tomo(s, a):
    d = tempfile.mkdtemp(prefix="moao_case_")
    P.write_system(d, s, a, profile_names=("prof-1-atmos-night0.txt",))
    return M.Tomo(os.path.join(d, "sys-params.txt"), os.path.join(d, "prof-1-atmos-night0.txt"))


def _empty(rows, cols):
    """A column-major rows x cols matrix (held as its transpose)."""
    return torch.zeros((cols, rows), dtype=F64, device=DEV)


# --------------------------------------- Matern-5/2 slope covariances (inputs)
_LAYERS = ((0.0, 0.55, 3.0), (4000.0, 0.3, 4.0), (11000.0, 0.15, 5.0))  # altitude, weight, scale / pitch
_SIGNAL, _NOISE, _LGS = 0.0137, 1.0e-4, 0.1


def _slopes(s, m, n, x, y, weights, projected=True):
    """2N x 2N slope covariance of WFS m against WFS n (rows m, columns n)."""
    N = x.numel()
    out = torch.zeros((2 * N, 2 * N), dtype=F64, device=DEV)
    for (h, _, scale), wt in zip(_LAYERS, weights):
        if projected:
            (xm, ym), (xn, yn) = _projected(s, m, h, x, y), _projected(s, n, h, x, y)
        else:
            (xm, ym), (xn, yn) = (x, y), (x, y)
        a = math.sqrt(5.0) / (scale * s.diam / s.nssp)
        du, dv = xm[:, None] - xn[None, :], ym[:, None] - yn[None, :]
        r = a * torch.sqrt(du * du + dv * dv)
        e = torch.exp(-r) * (_SIGNAL * wt)
        r = e * (1.0 + r)
        du, dv = a * du, a * dv
        out[:N, :N] += r - e * du * du
        out[N:, N:] += r - e * dv * dv
        xy = e * du * dv
        out[:N, N:] -= xy
        out[N:, :N] -= xy
    return out


def _weights(seed):
    g = np.random.default_rng(seed)
    w = np.array([l[1] for l in _LAYERS]) * g.lognormal(0.0, 0.3, len(_LAYERS))
    return (w / w.sum()).tolist()


def _noise(s, seed, nmeas):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 77)
    return _NOISE * (1.0 + 2.0 * torch.rand(nmeas, generator=g, dtype=F64, device=DEV))


def _model_cmm(s, seed):
    """Cmm, lower triangle, column-major (as its transpose: row j = column j)."""
    x, y = _centres(s)
    N2 = 2 * x.numel()
    nw = s.nW - 1
    w = _weights(seed)
    C = _empty(N2 * nw, N2 * nw)
    for n in range(nw):
        for m in range(n, nw):
            b = _slopes(s, m, n, x, y, w)
            if m == n and m < s.nLgs:
                b[:N2 // 2, :N2 // 2] += _LGS
                b[N2 // 2:, N2 // 2:] += _LGS
            C[n * N2:(n + 1) * N2, m * N2:(m + 1) * N2] = (b.tril() if m == n else b).t()
            del b
    C.diagonal().add_(_noise(s, seed, N2 * nw))
    return C


def _model_ctm(s, seed, shift_as=0.0):
    """Ctm (truth sensor rows), column-major; shift_as moves the target off axis."""
    x, y = _centres(s)
    N2 = 2 * x.numel()
    nw = s.nW - 1
    w = _weights(seed)
    ax = s.alphaX_as[nw]
    s.alphaX_as[nw] = ax + shift_as
    T = _empty(N2, N2 * nw)
    for n in range(nw):
        T[n * N2:(n + 1) * N2] = _slopes(s, nw, n, x, y, w).t()
    s.alphaX_as[nw] = ax
    return T


def _offsets(s, nmeas):
    N = nmeas // (2 * (s.nW - 1))
    b = [N * k for k in range(2 * s.nLgs)]
    return b, [v + N for v in b], [_LGS] * len(b)


def _sym(C):
    return torch.tril(C.t()) + torch.tril(C.t(), -1).t()


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "cov":
        s, a = _system(case, seed)
        t = _tomo(s, a)
        t.setTarget(0)
        nm, nts = t.getNMeas(), t.getNMeasTS()
        return {"case": case, "t": t, "nm": nm, "nts": nts, "cn2": np.array(a.cn2),
                "h": np.array(a.h), "L0": np.array(a.L0), "Cmm": _empty(nm, nm),
                "Ctm": _empty(nts, nm), "Ctt": _empty(nts, nts), "ctx": _context()}
    if kind == "rec":
        s, _ = _system(case, seed)
        Cmm = _model_cmm(s, seed)
        nm = Cmm.shape[0]
        Ctm = torch.stack([_model_ctm(s, seed, 20.0 * g) for g in range(case["ngal"])])
        return {"case": case, "nm": nm, "nts": Ctm.shape[2], "Cmm": Cmm, "Ctm": Ctm,
                "R": torch.empty_like(Ctm), "off": _offsets(s, nm), "ctx": _context()}
    if kind == "cee":
        s, _ = _system(case, seed)
        Cmm = _model_cmm(s, seed)
        nm = Cmm.shape[0]
        Ctm = _model_ctm(s, seed)
        nts = Ctm.shape[1]
        x, y = _centres(s)
        Ctt = _slopes(s, s.nW - 1, s.nW - 1, x, y, _weights(seed), projected=False)
        L = torch.linalg.cholesky(_sym(Cmm))
        R = torch.cholesky_solve(Ctm, L)  # column-major R = Ctm Cmm^-1
        del L
        nact = I.make_dm(case["nssp"], 0.2, s.obs).nactu
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed))
        Dx = torch.randn((nts, nact), generator=g, dtype=F64, device=DEV)
        return {"case": case, "nm": nm, "nts": nts, "nact": nact, "Cmm": Cmm, "Ctm": Ctm, "Ctt": Ctt,
                "R": R.contiguous(), "Dx": Dx, "Cpp": torch.empty_like(Ctt),
                "Cpm": torch.empty_like(Ctm), "Cee": _empty(nts, nts), "Cvv": _empty(nact, nact),
                "Tmp": _empty(nact, nts), "off": _offsets(s, nm), "ctx": _context()}
    if kind == "psf":
        ins = I.intersample_inputs(case["nssp"], 39.0, 0.28)
        isx = M.Intersample(ins.nact ** 2, ins.np_, 39.0, ins.idx, ins.abs2fi, ins.otf, ctx=_context())
        return {"case": case, "isx": isx, "Cvv": _model_cvv(ins, seed)}
    tomos = [_tomo(s, a) for s, a in _survey(case, seed)]
    outs = [torch.zeros(t.getNMeas() * t.getNMeasTS(), dtype=F64, device=DEV) for t in tomos]
    return {"case": case, "tomos": tomos, "outs": outs, "ctx": _context()}


def _model_cvv(ins, seed):
    """Actuator covariance of a partly corrected wavefront: an exponential of the
    actuators' distance, at the amplitude of a Strehl ratio near one half."""
    g = np.random.default_rng(int(seed))
    p = torch.from_numpy(np.stack([ins.dm.csX, ins.dm.csY], 1)).to(DEV)
    d = torch.cdist(p, p)
    return (g.uniform(0.5, 1.5) * 0.01) * torch.exp(-d * g.uniform(4.0, 8.0))


# ----------------------------------------------------------------------- run
def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "cov":
        t, nm, nts, ctx = st["t"], st["nm"], st["nts"], st["ctx"]
        t.set_profile(st["cn2"], st["h"], st["L0"])
        M.matcov_tile(st["Cmm"], nm, nm, 0, 0, nm, t, 1, ctx=ctx)
        M.matcov_tile(st["Ctm"], nts, nm, 0, 0, nts, t, 3, ctx=ctx)
        M.matcov_tile(st["Ctt"], nts, nts, 0, 0, nts, t, 4, ctx=ctx)
        return {"Cmm": st["Cmm"], "Ctm": st["Ctm"], "Ctt": st["Ctt"]}
    if kind == "rec":
        nm, nts, ctx = st["nm"], st["nts"], st["ctx"]
        work = _work_buffer(st["Cmm"])
        work.copy_(st["Cmm"])
        st["R"].copy_(st["Ctm"])
        ctx.set_offsets(*(st["off"] if case["prec"] == "mixed" else ([], [], [])))
        M.reconstructor(nm, nts, work, nm, st["R"], nts, case["ngal"], prec=case["prec"], ctx=ctx)
        return {"R": st["R"], "L": work}
    if kind == "cee":
        nm, nts, na, ctx = st["nm"], st["nts"], st["nact"], st["ctx"]
        st["Cpp"].copy_(st["Ctt"])
        st["Cpm"].copy_(st["Ctm"])
        ctx.set_offsets(*(st["off"] if case["prec"] == "mixed" else ([], [], [])))
        M.Cee_Cvv(nm, nts, na, st["Cmm"], nm, st["Cpp"], nts, st["Cpm"], nts, st["R"], nts, st["Dx"],
                  na, st["Cee"], nts, st["Cvv"], na, st["Tmp"], na, prec=case["prec"], ctx=ctx)
        return {"Cee": st["Cee"], "Cvv": st["Cvv"], "RCmm": st["Cpm"]}
    if kind == "psf":
        return st["isx"].process(st["Cvv"])
    per, _ = B.batch_reconstructors(st["tomos"], st["outs"], prec=case["prec"],
                                    packed_max=case["packed"], ctx=st["ctx"])
    return {"R": st["outs"], "status": [p["status"] for p in per]}


_WORK = {}


def _work_buffer(like):
    """The buffer that the factor overwrites: one per program, not per system."""
    n = like.numel()
    if _WORK.get("n") != n:
        _WORK.clear()
        _WORK.update(n=n, buf=torch.empty_like(like))
    return _WORK["buf"]


# --------------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "cov":
        s, a = _system(case, seed)
        if _sizes(case)[0] ** 2 * a.nLayer > 4e9:
            return None
        return {"Cmm": torch.tril(_cmm(s, a)).t(), "Ctm": _ctm(s, a).t(), "Ctt": _ctt(s, a).t()}
    if kind == "rec":
        s, _ = _system(case, seed)
        Cmm = _model_cmm(s, seed)
        Ctm = torch.stack([_model_ctm(s, seed, 20.0 * g) for g in range(case["ngal"])])
        L = torch.linalg.cholesky(_sym(Cmm))
        del Cmm
        R = torch.stack([torch.cholesky_solve(T, L) for T in Ctm])
        # the mixed path leaves the FP32 factor of Cmm less the declared constants
        return {"R": R, "L": L.t() if case["prec"] == "fp64" else None}
    if kind == "cee":
        st = prepare(case, seed)
        Cs, Cm, R, Dx = _sym(st["Cmm"]), st["Ctm"].t(), st["R"].t(), st["Dx"].t()
        RC = R @ Cs
        del Cs
        CR = Cm @ R.t()
        Cee = st["Ctt"].t() - CR - CR.t() + RC @ R.t()
        return {"Cee": Cee.t(), "Cvv": (Dx @ Cee @ Dx.t()).t(), "RCmm": RC.t()}
    if kind == "psf":
        ins = I.intersample_inputs(case["nssp"], 39.0, 0.28)
        return _psf(_model_cvv(ins, seed), ins)
    R = []
    for s, a in _survey(case, seed):
        C = _cmm(s, a)
        C = torch.tril(C) + torch.tril(C, -1).t()
        X = torch.cholesky_solve(_ctm(s, a).t().contiguous(), torch.linalg.cholesky(C))
        R.append(X.reshape(-1))  # (nmeas, nmeasts) row-major = R column-major
    return {"R": R, "status": [0] * case["count"]}


_GA = (0, 12.067619015983075, 5.17183672113560444, 0.795667187867016068, 0.0628158306210802181,
       0.00301515986981185091, 9.72632216068338833e-05, 2.25320204494595251e-06,
       3.93000356676612095e-08, 5.34694362825451923e-10, 5.83302941264329804e-12)
_GMA = (-3.74878707653729304, -2.04479295083852408, -0.360845814853857083, -0.0313778969438136685,
        -0.001622994669507603, -5.56455315259749673e-05, -1.35720808599938951e-06,
        -2.47515152461894642e-08, -3.50257291219662472e-10, -3.95770950530691961e-12,
        -3.65327031259100284e-14)
_K1, _K2, _K3 = 0.1716613621245709486, 1.00563491799858928388289314170833, 1.25331413731550012081
_LAMBDA2 = 0.00026942094446267851


def _dphi(x, y, L0):
    """von Karman phase structure function of a separation (x, y)."""
    r = torch.sqrt(x * x + y * y) * (2 * math.pi / L0)
    z = 0.25 * r * r
    pg, pa = torch.full_like(z, _GMA[10]), torch.full_like(z, _GA[10])
    for k in range(9, -1, -1):
        pg = pg * z + _GMA[k]
    for k in range(9, 0, -1):
        pa = pa * z + _GA[k]
    near = -0.5 * (r ** (5.0 / 3.0) * pg + z * pa)
    i = 1.0 / r.clamp_min(1.0)
    far = _K2 - _K3 * torch.exp(-r) * r ** (1.0 / 3.0) * (
        1.0 + i * (0.22222222222222222222 + i * (-0.08641975308641974829 + i * 0.08001828989483310284)))
    return torch.where(r > 1.5 * math.pi, far, near) * (_K1 * L0 ** (5.0 / 3.0))


def _stencils(du, dv, s1, s2, L0):
    """Slope covariances xx, xy, yx, yy of subapertures of half sizes s1, s2."""
    D = lambda p, q: _dphi(du + p, dv + q, L0)  # noqa: E731
    c, d = s1 - s2, s1 + s2
    return (-D(c, 0) + D(d, 0) + D(-d, 0) - D(-c, 0), -D(s1, -s2) + D(s1, s2) + D(-s1, -s2) - D(-s1, s2),
            -D(-s2, s1) + D(s2, s1) + D(-s2, -s1) - D(s2, -s1), -D(0, c) + D(0, d) + D(0, -d) - D(0, -c))


def _block(s, a, m, n, projected=True):
    x, y = _centres(s)
    N = x.numel()
    ssp = s.diam / s.nssp
    out = torch.zeros((2 * N, 2 * N), dtype=F64, device=DEV)
    for cn2, h, L0 in zip(a.cn2, a.h, a.L0):
        if projected:
            (xm, ym), (xn, yn) = _projected(s, m, h, x, y), _projected(s, n, h, x, y)
            sm, sn = ssp * (1.0 - s.gsAlt[m] * h), ssp * (1.0 - s.gsAlt[n] * h)
        else:
            (xm, ym), (xn, yn), sm, sn = (x, y), (x, y), ssp, ssp
        if not (sm > 0 and sn > 0):
            continue
        f = 0.5 * _LAMBDA2 / (ssp * ssp) * cn2
        xx, xy, yx, yy = _stencils(xm[:, None] - xn[None], ym[:, None] - yn[None], sm / 2, sn / 2, L0)
        out[:N, :N] += f * xx
        out[:N, N:] += f * xy
        out[N:, :N] += f * yx
        out[N:, N:] += f * yy
    return out


def _photons(mag, throughput, d, tframe, bdw):
    """Photons per subaperture and frame of an NGS of this magnitude."""
    return 10 ** (2.9 - 0.4 * mag) * throughput * d * d * tframe * bdw * 1e4


def _wfs_noise(s, a):
    """(NGS variance per NGS, LGS xx, yy, xy per LGS): the photometric noise."""
    r0 = float(sum(a.cn2)) ** (-3.0 / 5.0)
    see = lambda lam: (5e-7 / r0 * (5e-7 / lam) ** 0.2 * RASC) ** 2  # noqa: E731
    d = s.diam / s.nssp
    ngs = []
    for k in range(s.nNgs):
        F = _photons(s.mrNGS[k], s.throughNGS, d, s.tFrame, s.bdw_m * 1e10)
        e = see(s.lambdaNGS)
        ngs.append(0.32 / F * e + 0.82 * (s.RON / (F * s.ngsPixSize)) ** 2 * e * e)
    lgs = []
    x, y = _centres(s)
    F = s.lgsFlux * s.tFrame * d * d * s.throughLGS / s.throughAtm
    for w in range(s.nLgs):
        ax, ay = s.alphaX_as[w] / RASC, s.alphaY_as[w] / RASC
        nrm = math.sqrt(ax * ax + ay * ay)
        lx, ly = ax * s.diam / 2 / nrm, ay * s.diam / 2 / nrm
        fw = RASC * s.lgsDepth / (s.lgsAlt * s.lgsAlt)
        e2 = ((x - lx) ** 2 + (y - ly) ** 2) * fw * fw
        th = torch.atan2(y - ly, x - lx)
        pe = see(s.lambdaLGS) + s.spotWidth ** 2
        f1, f2 = 0.32 / F, 0.82 * (s.RON / (F * s.lgsPixSize)) ** 2
        short = f1 * pe + f2 * pe * pe
        long_ = f1 * (pe + e2) + f2 * (pe + e2) ** 1.5 * pe ** 0.5
        c, si = torch.cos(th), torch.sin(th)
        lgs.append((long_ * c * c + short * si * si, long_ * si * si + short * c * c,
                    (long_ - short) * si * c))
    return ngs, lgs


def _cmm(s, a):
    """Lower blocks of Cmm (blocks above the diagonal left 0)."""
    nw = s.nW - 1
    ngs, lgs = _wfs_noise(s, a)
    N2 = 2 * _centres_count(s)
    N = N2 // 2
    C = torch.zeros((N2 * nw, N2 * nw), dtype=F64, device=DEV)
    for m in range(nw):
        for n in range(m + 1):
            b = _block(s, a, m, n)
            if m == n and m < s.nLgs:
                for k, (p, q) in enumerate(((0, 0), (N, N), (N, 0), (0, N))):
                    b[p:p + N, q:q + N].diagonal().add_(lgs[m][min(k, 2)])
                    if p == q:
                        b[p:p + N, q:q + N] += s.lgsCst
            elif m == n:
                b.diagonal().add_(ngs[m - s.nLgs])
            C[m * N2:(m + 1) * N2, n * N2:(n + 1) * N2] = b
    return C


def _ctm(s, a):
    on_axis = list(s.alphaX_as), list(s.alphaY_as)
    s.alphaX_as[-1], s.alphaY_as[-1] = s.targetX_as[0], s.targetY_as[0]
    T = torch.cat([_block(s, a, s.nW - 1, n) for n in range(s.nW - 1)], 1)
    s.alphaX_as, s.alphaY_as = on_axis
    return T


def _ctt(s, a):
    return _block(s, a, s.nW - 1, s.nW - 1, projected=False)


def _psf(Cvv, ins):
    n = ins.np_
    N = int(max(512, 8 * 2 ** int(math.log(n) + 0.5)))
    dp = N // (3 * (n - 1)) + 1
    nc = 2 * n - 1
    idx = torch.from_numpy(ins.idx).to(DEV) - 1
    m = torch.zeros(nc * nc, dtype=F64, device=DEV).index_add_(0, idx, Cvv.t().reshape(-1))
    hits = torch.bincount(idx, minlength=nc * nc)
    m = m / hits.clamp_min(1)
    a = N // 2 - (nc - 1) // 2 * dp
    grid = torch.zeros((N, N), dtype=F64, device=DEV)
    grid[a:a + nc * dp:dp, a:a + nc * dp:dp] = m.reshape(nc, nc)
    A2 = torch.from_numpy(ins.abs2fi).to(DEV)
    O2 = torch.from_numpy(ins.otf).to(DEV)
    H = N // 2 + 1
    half = lambda v: torch.fft.irfft2(v.to(torch.complex128), s=(N, N)) * (N * N)  # noqa: E731
    dphi = half(torch.fft.rfft2(grid).real * A2.t()[:, :H])
    k = 2 * (2 * 3.14159 / 1.65e-06) ** 2 / (N * N * float(dp) * float(dp))
    dphi = torch.exp(-0.5 * (dphi[N // 2, N // 2] * k - dphi * k))
    dphi = torch.roll(dphi, (N // 2, N // 2), (0, 1))
    return torch.roll(half((O2 * dphi).t()[:, :H]), (N // 2, N // 2), (0, 1))


# ---------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "psf":
        na = I.make_dm(case["nssp"], 0.2, 0.28).nactu
        N = 512
        fft = 5.0 * N * N * math.log2(N * N) / 2  # a real 2-D transform
        return {"bytes": 8.0 * (na * na + 3 * N * N), "flops": 3 * fft}
    if kind == "batch":
        b = f = 0.0
        for s, _ in _survey(case, 1):
            m = 2.0 * _centres_count(s)
            n = m * (s.nW - 1)
            b += 8 * m * n
            f += n ** 3 / 3 + 2 * m * n * n
        return {"bytes": b, "flops": f}
    n, m = (float(v) for v in _sizes(case))
    if kind == "cov":
        # ~45 operations per structure-function value; pairs of guide stars at
        # unequal altitudes need four values per subaperture pair and layer,
        # the others are functions of the grid offset
        N = m / 2
        unequal = case["nlgs"] * (case["nngs"] + 1) if case["system"] == "39m" else 6
        return {"bytes": 8 * (n * (n + 1) / 2 + m * n + m * m),
                "flops": 45.0 * 4 * unequal * N * N * case["nlayer"]}
    if kind == "rec":
        g = case["ngal"]
        return {"bytes": 8 * (n * n + 2 * g * m * n), "flops": n ** 3 / 3 + 2 * g * m * n * n}
    na = float(I.make_dm(case["nssp"], 0.2, 0.28).nactu)
    return {"bytes": 8 * (n * n / 2 + 3 * m * n + 2 * m * m + na * m + na * na),
            "flops": 2 * m * n * n + 4 * m * m * n + 2 * na * m * m + 2 * na * na * m}
