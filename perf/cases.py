"""What is measured of this framework: the calls its users make, over the range they make them in.

Every case runs public entry points only: P(k) and sources from the perturbation solver (one mode to
thousands, one cosmology to many, both precisions, small and large hierarchies, default and tight
tolerances), the full C_l pipeline (solver -> k-interpolation -> line of sight -> C_l), the same
pipeline on sources the caller already has, the stand-alone line-of-sight and k-integral calls on
host arrays, the spherical Bessel cache, and the source surrogate's network (training and
inference).  Parameters, sources and weights come from the seed; grid sizes from the case.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "symboltz.jl_gb300"))

import symboltz as S  # noqa: E402
from symboltz.surrogate import MLP  # noqa: E402

HMPC = 299792458.0 / 1e5  # k in h/Mpc -> H0/c


def listed():
    return [
        # a handful of modes of the reference's small test model: the smallest useful call (latency)
        dict(name="pk_few", kind="pk", lmax_g=5, lmax_nu=5, lmax_h=5, nx=4, precision="mixed", rtol=1e-5, atol=1e-5, ncosmo=1, nk=4,
             kmin=3e-4, kmax=0.3),
        # P(k) of one cosmology with the library's default model and tolerances
        dict(name="pk_default", kind="pk", lmax_g=10, lmax_nu=10, lmax_h=10, nx=4, precision="mixed", rtol=1e-5, atol=1e-5, ncosmo=1,
             nk=100, kmin=1e-4, kmax=1.0),
        # plain LCDM (massless neutrinos) in all-FP64 arithmetic, as a precision run
        dict(name="pk_plain_fp64", kind="pk", lmax_g=10, lmax_nu=10, lmax_h=10, nx=0, precision="fp64", rtol=1e-6, atol=1e-6, ncosmo=1,
             nk=100, kmin=1e-4, kmax=1.0),
        # a parameter study: many cosmologies with ragged k grids solved in one launch
        dict(name="pk_batch", kind="pk", lmax_g=30, lmax_nu=10, lmax_h=10, nx=5, precision="mixed", rtol=1e-5, atol=1e-5, ncosmo=24,
             nk=256, kmin=1e-4, kmax=0.2),
        # perturbation factors on a (k, tau) grid: a shard of the surrogate's training set
        dict(name="factors_shard", kind="factors", lmax_g=10, lmax_nu=10, lmax_h=10, nx=5, precision="mixed", rtol=1e-5, atol=1e-5,
             ncosmo=6, nk=61, ntau=301, kmin=1e-4, kmax=0.3),
        # the C_l driver with its default grids (Chebyshev k grid, 300 times), temperature, E and lensing
        dict(name="cmb_default", kind="cmb", lmax_g=5, lmax_nu=5, lmax_h=5, nx=4, rtol=1e-5, atol=1e-5, skip=-1.0, modes="TT EE ψψ",
             grid="default", nk=0, ntau=300, nl=200, lmax=2500, kmin=0.0, kmax=0.0),
        # the headline spectrum: massive neutrino, photon l_max 30, 1000 k, 2000 tau, TT/TE/EE to l = 2500
        dict(name="cmb_headline", kind="cmb", lmax_g=30, lmax_nu=10, lmax_h=10, nx=5, rtol=1e-6, atol=3e-8, skip=1e-2, modes="TT TE EE",
             grid="spline", nk=1000, ntau=2000, nl=200, lmax=2500, kmin=1e-5, kmax=5.0),
        # C_l from sources in hand (the surrogate's path): k-interpolation, line of sight, k-integral
        dict(name="cmb_sources", kind="cmb_sources", los="mixed", modes="TT TE EE", nk=400, ntau=500, nl=200, lmax=2500, kmin=1e-4,
             kmax=0.5),
        # the line-of-sight and k-integral calls on the caller's own source arrays (FP64)
        dict(name="los_cl", kind="los", nsrc=2, nk=777, ntau=401, nl=97, lmax=1500, kmax=1800.0),
        # the Bessel table a program builds once per set of multipoles, and reads of it
        dict(name="bessel_2500", kind="bessel", nl=200, lmax=2500, nx=20000, hermite=True),
        # training steps of the source surrogate's network at its batch size
        dict(name="mlp_train", kind="mlp_train", nin=10, width=512, nhidden=4, nout=7, batch=65536, rows=300000, steps=16),
        # the network evaluated on one cosmology's (k, tau) grid
        dict(name="mlp_infer", kind="mlp_infer", nin=10, width=512, nhidden=4, nout=7, batch=65536, rows=200000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _logi(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def draw(rng):
    kind = rng.choice(["pk", "pk", "pk", "batch", "factors", "cmb", "cmb_sources", "los", "bessel", "mlp_train", "mlp_infer"])
    if kind in ("pk", "batch", "factors", "cmb"):
        m = dict(lmax_g=rng.choice([4, 5, 8, 10, 13, 17, 30]), lmax_nu=rng.choice([4, 5, 8, 10, 17]), lmax_h=rng.choice([4, 5, 8, 10]),
                 nx=rng.choice([0, 3, 4, 5]))
    if kind == "pk":
        tol = rng.choice([1e-5, 1e-5, 1e-6])
        return dict(kind="pk", **m, precision=rng.choice(["mixed", "mixed", "fp64"]), rtol=tol, atol=tol, ncosmo=1, nk=_logi(rng, 1, 600),
                    kmin=_log(rng, 1e-5, 1e-3), kmax=_log(rng, 0.05, 2.0))
    if kind == "batch":
        return dict(kind="pk", **m, precision=rng.choice(["mixed", "mixed", "mixed", "fp64"]), rtol=1e-5, atol=1e-5,
                    ncosmo=rng.randint(2, 24), nk=_logi(rng, 40, 256), kmin=1e-4, kmax=_log(rng, 0.05, 0.2))
    if kind == "factors":
        return dict(kind="factors", **m, precision="mixed", rtol=1e-5, atol=1e-5, ncosmo=rng.randint(1, 6), nk=_logi(rng, 10, 100),
                    ntau=_logi(rng, 20, 500), kmin=1e-4, kmax=_log(rng, 0.05, 0.3))
    if kind == "cmb":
        if rng.random() < 0.5:
            return dict(kind="cmb", **m, rtol=1e-5, atol=1e-5, skip=-1.0, modes=rng.choice(["TT", "TT TE EE", "TT EE ψψ"]), grid="default",
                        nk=0, ntau=rng.randint(150, 500), nl=rng.randint(40, 200), lmax=rng.randint(500, 2500), kmin=0.0, kmax=0.0)
        return dict(kind="cmb", **m, rtol=1e-6, atol=1e-6, skip=1e-2, modes="TT TE EE", grid="spline", nk=_logi(rng, 150, 1000),
                    ntau=_logi(rng, 300, 2000), nl=rng.randint(50, 200), lmax=rng.randint(800, 2500), kmin=1e-4, kmax=_log(rng, 0.2, 1.0))
    if kind == "cmb_sources":
        return dict(kind="cmb_sources", los=rng.choice(["mixed", "mixed", "fp64"]), modes=rng.choice(["TT", "TT TE EE"]),
                    nk=_logi(rng, 60, 400), ntau=_logi(rng, 120, 700), nl=rng.randint(30, 200), lmax=_logi(rng, 400, 2500), kmin=1e-4,
                    kmax=_log(rng, 0.2, 0.6))
    if kind == "los":
        return dict(kind="los", nsrc=rng.randint(1, 3), nk=_logi(rng, 60, 1000), ntau=_logi(rng, 50, 600), nl=_logi(rng, 5, 150),
                    lmax=_logi(rng, 200, 2000), kmax=_log(rng, 150.0, 2000.0))
    if kind == "bessel":
        return dict(kind="bessel", nl=_logi(rng, 10, 200), lmax=_logi(rng, 300, 2500), nx=_logi(rng, 100, 20000),
                    hermite=rng.choice([True, True, False]))
    net = dict(nin=rng.choice([7, 8, 10]), width=rng.choice([128, 256, 512]), nhidden=rng.randint(2, 4), nout=rng.choice([1, 4, 7]))
    if kind == "mlp_train":
        return dict(kind="mlp_train", **net, batch=rng.choice([4096, 8192, 32768, 65536]), rows=_logi(rng, 50000, 300000),
                    steps=rng.randint(3, 16))
    return dict(kind="mlp_infer", **net, batch=rng.choice([8192, 65536]), rows=_logi(rng, 128, 300000))


# ---- inputs ----------------------------------------------------------------------------------
def _pars(rng, massive):
    """Parameters near the Planck values."""
    h = rng.uniform(0.64, 0.71)
    p = dict(h=h, Omega_c=rng.uniform(0.115, 0.125) / h**2, Omega_b=rng.uniform(0.0216, 0.0228) / h**2, T0=2.7255,
             Neff=2.0328 if massive else 3.046, YHe=0.245, ln_As1e10=rng.uniform(3.0, 3.1), ns=rng.uniform(0.95, 0.98), m_nu_eV=0.0,
             N_nu=0.0)
    if massive:
        p.update(m_nu_eV=rng.uniform(0.06, 0.2), N_nu=1.0)
    return p


def _model(case):
    return S.ΛCDM(lmax_gamma=case["lmax_g"], lmax_nu=case["lmax_nu"], lmax_h=case["lmax_h"], nx=max(1, case["nx"]),
                  massive_nu=case["nx"] > 0)


def _ragged(case):
    """Modes per cosmology: nk, or ragged around nk where there are several cosmologies."""
    n = case["ncosmo"]
    if n == 1:
        return [case["nk"]]
    return [int(v) for v in np.random.default_rng(case["nk"]).integers(max(2, case["nk"] // 2), case["nk"] * 3 // 2 + 1, size=n)]


def _kgrid(case, n):
    if n == 1:
        return np.array([math.sqrt(case["kmin"] * case["kmax"]) * HMPC])
    return np.geomspace(case["kmin"], case["kmax"], n) * HMPC


def _ls(case):
    return np.unique(np.round(np.geomspace(2, case["lmax"], case["nl"])).astype(np.int32))


def _tau0(p):
    """Conformal age of a massless-neutrino LCDM universe in 1/H0."""
    og = 2.47282e-5 / p["h"] ** 2
    orad = og * (1 + p["Neff"] * 7 / 8 * (4 / 11) ** (4 / 3))
    om = p["Omega_c"] + p["Omega_b"]
    x, w = np.polynomial.legendre.leggauss(200)
    u = 0.5 * (x + 1)  # a = u^2
    a = u * u
    return float(np.sum(0.5 * w * 2 * u / np.sqrt(orad + om * a + (1 - orad - om) * a**4)))


def _line_sources(rng, ks, taus, nsrc):
    """Sources with the shape the path meets: a recombination peak carrying Silk-damped acoustic
    oscillations in k, and a smooth late-time part.  [nk][ntau][nsrc], zero at the last time."""
    k, t = ks[:, None], taus[None, :]
    kd = rng.uniform(350, 420)
    rs = rng.uniform(0.033, 0.036)
    vis = np.exp(-0.5 * ((t - 0.063) / rng.uniform(0.0028, 0.0034)) ** 2) * 120
    out = np.zeros((len(ks), len(taus), nsrc))
    damp = np.exp(-((k / kd) ** 1.4))
    a = rng.uniform(0.5, 1.5, size=(3, 4))
    for s in range(nsrc):
        osc = a[s, 0] * np.cos(k * rs * (t / 0.063)) + 0.5 * a[s, 1] * np.sin(k * rs * (t / 0.063)) + 0.1 * a[s, 2]
        late = 0.05 * a[s, 3] * np.exp(-t) / (1 + (k * 0.02) ** 2)
        out[:, :, s] = k * (vis * osc * damp + late) / (1 + s * k * 0.01)
    out[:, -1, :] = 0
    return out


def _net_params(case, rng):
    sizes = [case["nin"]] + [case["width"]] * case["nhidden"] + [case["nout"]]
    p = []
    for a, b in zip(sizes[:-1], sizes[1:]):
        p.append(rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / (a + b)))
        p.append(rng.uniform(-0.05, 0.05, b))
    return sizes, np.concatenate(p).astype(np.float32)


def _net_data(case, rng):
    X = rng.uniform(-1, 1, (case["rows"], case["nin"])).astype(np.float32)
    F = rng.normal(size=(case["nin"], case["nout"]))
    Y = (np.sin(2 * X @ F) + 0.05 * rng.normal(size=(case["rows"], case["nout"]))).astype(np.float32)
    return X, Y


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = dict(case=dict(case))
    if kind in ("pk", "factors"):
        prob = S.CosmologyProblem(_model(case), [_pars(rng, case["nx"] > 0) for _ in range(case["ncosmo"])], precision=case["precision"],
                                  pt_rtol=case["rtol"], pt_atol=case["atol"])
        bg = prob.solvebg()
        ns = _ragged(case)
        st.update(prob=prob, ks=np.concatenate([_kgrid(case, n) for n in ns]), cosmo=np.repeat(np.arange(len(ns)), ns))
        if kind == "factors":
            st["taus"] = np.stack([0.01 + (t0 - 0.01) * S.cosgrid(0.0, 1.0, length=case["ntau"]) for t0 in bg.tau0])
    elif kind == "cmb":
        M = _model(case)
        opts = {} if case["skip"] < 0 else dict(refine_skip=case["skip"])
        prob = S.CosmologyProblem(M, _pars(rng, case["nx"] > 0), pt_rtol=case["rtol"], pt_atol=case["atol"], **opts)
        bg = prob.solvebg()
        ls = _ls(case)
        st.update(prob=prob, pars=prob.pars[0], jl=S.SphericalBesselCache(ls, xmax=20.0 * 2500), lall=np.arange(2, int(ls[-1]) + 1),
                  modes=case["modes"].split(" "), kw={})
        if case["grid"] == "spline":
            st["kw"] = dict(kinterp=S.CubicSplineInterpolator(np.geomspace(case["kmin"], case["kmax"], case["nk"]) * HMPC, f=np.log))
        st["kw"]["xs"] = S.cosgrid(0.0, 1.0, length=case["ntau"])
        del bg
    elif kind == "cmb_sources":
        prob = S.CosmologyProblem(S.ΛCDM(lmax=5, massive_nu=False), _pars(rng, False), los_precision=case["los"])
        prob.solvebg()
        t0 = _tau0(prob.pars[0])
        ks = np.geomspace(case["kmin"], case["kmax"], case["nk"]) * HMPC
        taus = 0.01 + (t0 - 0.01) * (1 - np.cos(np.pi * np.linspace(0, 0.5, case["ntau"])))
        ls = _ls(case)
        st.update(prob=prob, jl=S.SphericalBesselCache(ls), lall=np.arange(2, int(ls[-1]) + 1), modes=case["modes"].split(" "),
                  kinterp=S.CubicSplineInterpolator(ks, f=np.log), taus=taus, sources=_line_sources(rng, ks, taus, 3))
    elif kind == "los":
        t0 = 3.2
        ks = np.linspace(case["kmax"] / case["nk"], case["kmax"], case["nk"])
        taus = 0.01 + (t0 - 0.01) * (1 - np.cos(np.pi * np.linspace(0, 0.5, case["ntau"])))
        ls = _ls(case)
        src = _line_sources(rng, ks, taus, case["nsrc"])
        P0 = 2 * np.pi**2 * 2.1e-9 / ks**3 * (ks / 100.0) ** (-0.035)
        st.update(ls=ls, ks=ks, taus=taus, P0=P0, S=np.ascontiguousarray(src.transpose(1, 0, 2)),
                  jl=S.SphericalBesselCache(ls, xmax=max(20.0 * int(ls[-1]), 1.01 * t0 * case["kmax"])))
    elif kind == "bessel":
        ls = _ls(case)
        xmax = 20.0 * int(ls[-1])
        st.update(ls=ls, xs=rng.uniform(0.0, xmax, case["nx"]), at=sorted({0, len(ls) // 3, len(ls) // 2, len(ls) - 1}))
    else:
        _, p = _net_params(case, rng)
        X, Y = _net_data(case, rng)
        net = MLP(case["nin"], case["width"], case["nhidden"], case["nout"], case["batch"], 1)
        net.set_params(p)
        st.update(net=net, X=X)
        if kind == "mlp_train":
            net.set_data(X, Y)
    return st


# ---- one pass --------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "pk":
        P, status = S.spectrum_matter(st["prob"], st["ks"], cosmo=st["cosmo"], return_status=True)
        return {"P": P, "status": status}
    if kind == "factors":
        F, status, steps = S.solvept(st["prob"], st["ks"], 1e-6, saveat=st["taus"], output="factors", cosmo=st["cosmo"])
        return {"factors": F, "status": status}
    if kind == "cmb":  # a whole cosmology, as a sampler's likelihood call: new parameters, background, modes, C_l
        st["prob"].set_params(st["pars"])
        D, status = S.spectrum_cmb(st["modes"], st["prob"], st["jl"], st["lall"], normalization="Dl", return_status=True, **st["kw"])
        return {"Dl": D, "status": status}
    if kind == "cmb_sources":
        return {"Dl": S.spectrum_cmb(st["modes"], st["prob"], st["jl"], st["lall"], kinterp=st["kinterp"], taus=st["taus"],
                                     normalization="Dl", sources=st["sources"])}
    if kind == "los":
        Th = S.los_integrate(st["S"], st["ls"], st["taus"], st["ks"], st["jl"])
        A, B = np.ascontiguousarray(Th[:, :, 0]), np.ascontiguousarray(Th[:, :, -1])
        return {"Theta": Th, "Cl": S.spectrum_cmb(A, B, st["P0"], st["ls"], st["ks"])}
    if kind == "bessel":
        jl = S.SphericalBesselCache(st["ls"], hermite=case["hermite"])
        return {"j": np.stack([jl(il, st["xs"]) for il in st["at"]])}
    if kind == "mlp_train":
        loss = st["net"].train(case["steps"], 2e-4)
        return {"loss": loss, "params": st["net"].get_params()}
    return {"Y": st["net"].infer(st["X"])}


# ---- what a pass cannot do without -----------------------------------------------------------
def _nstate(case):
    n = 11 + 2 * (case["lmax_g"] - 2) + case["lmax_nu"] + 1
    return n + (case["nx"] * (case["lmax_h"] + 1) if case["nx"] else 0)


def _pt_flops(case, ks):
    """Right-hand sides and linear solves of an adaptive fifth-order Rosenbrock method with eight stages:
    a mode takes about 95 + 0.8 k tau0 steps, levelling off near 2000 at tolerance 1e-5 and rising to the
    full oscillation count at tighter ones; a step costs about 36 flops per unknown and stage (operator,
    stage sums, structured solve)."""
    x = 0.8 * 3.2 * np.asarray(ks)
    steps = 95 + x / (1 + x / 2400 * (case["atol"] / 1e-5) ** 0.6)
    return float(np.sum(steps)) * 8 * 36 * _nstate(case)


def work(case):
    kind = case["kind"]
    if kind in ("pk", "factors"):
        ks = np.concatenate([_kgrid(case, n) for n in _ragged(case)])
        nout = 1 if kind == "pk" else 7 * case["ntau"]
        return {"bytes": 8.0 * len(ks) * (1 + nout), "flops": _pt_flops(case, ks)}
    if kind in ("cmb", "cmb_sources"):
        nm = len(case["modes"].split(" "))
        ns = len(set(case["modes"].replace(" ", "")))
        if kind == "cmb" and case["grid"] == "default":
            ks = np.linspace(1e-2, 1e4, 131) if "ψ" in case["modes"] else np.linspace(1e-2, 2e3, 61)
        else:
            ks = np.geomspace(case["kmin"], case["kmax"], case["nk"]) * HMPC
        nl = len(_ls(case))
        nf = int((ks[-1] - ks[0]) * 3.2 / math.pi) + 2
        flops = nf * case["ntau"] * (12.0 * ns + nl * (8 + 2 * ns)) + 3.0 * nf * nl * nm
        nbytes = 8.0 * (nm * int(_ls(case)[-1]) + 3 * nf) + 8.0 * nl * min(20.0 * 2500, ks[-1] * 3.2) / (2 * math.pi / 15)
        if kind == "cmb":
            flops += _pt_flops(case, ks)
        else:
            nbytes += 8.0 * case["nk"] * case["ntau"] * ns
        return {"bytes": nbytes, "flops": flops}
    if kind == "los":
        nl = len(_ls(case))
        nk, nt, ns = case["nk"], case["ntau"], case["nsrc"]
        table = 16.0 * nl * 3.2 * case["kmax"] / (2 * math.pi / 15)
        return {"bytes": 8.0 * nk * (nt * ns + nl * ns) + table, "flops": nk * nt * nl * (8.0 + 2 * ns) + 10.0 * nk * nl}
    if kind == "bessel":
        nl, L = len(_ls(case)), int(_ls(case)[-1])
        n = 20.0 * L / (2 * math.pi / 15)
        return {"bytes": n * nl * (8.0 + (8.0 if case["hermite"] else 0.0) + 8.0) + 4 * 16.0 * case["nx"], "flops": n * L * 3.0}
    w, h = case["width"], case["nhidden"]
    p = case["nin"] * w + (h - 1) * w * w + w * case["nout"]
    if kind == "mlp_train":
        return {"bytes": case["steps"] * (case["batch"] * 4.0 * (case["nin"] + case["nout"]) + 28.0 * p),
                "flops": case["steps"] * 6.0 * case["batch"] * p}
    return {"bytes": 4.0 * case["rows"] * (case["nin"] + case["nout"]) + 4.0 * p, "flops": 2.0 * case["rows"] * p}


# ---- the same in 64 bits, without this repository's code ---------------------------------------
def _bessel_rows(ls, xmax, dx=2 * math.pi / 15):
    """j_l and j_l' on the cache's x grid, as float64 tensors [len(ls)][N + 1] (upward recurrence above
    the turning point, Miller's downward recurrence below), and the grid's spacing."""
    N = int(math.trunc(xmax / dx))
    step = xmax / (N - 1)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.arange(N, dtype=torch.float64, device=dev) * step
    x[-1] = xmax
    ls = [int(v) for v in ls]
    pos = {l: i for i, l in enumerate(ls)}
    L = ls[-1]
    y = torch.zeros((len(ls), N + 1), dtype=torch.float64, device=dev)
    dy = torch.zeros_like(y)
    up = torch.nonzero(x > L + 1)[:, 0]
    lo = torch.nonzero((x <= L + 1) & (x > 0))[:, 0]

    def start(xx):
        j0 = torch.sin(xx) / xx
        return j0, (j0 - torch.cos(xx)) / xx

    if len(up):
        xx = x[up]
        j0, j1 = start(xx)
        jm, jc, jn = torch.cos(xx) / xx, j0, j1
        for l in range(L + 1):
            if l in pos:
                y[pos[l], up] = jc
                dy[pos[l], up] = -jn if l == 0 else (l * jm - (l + 1) * jn) / (2 * l + 1)
            jm, jc, jn = jc, jn, (2 * l + 3) / xx * jn - jc
    if len(lo):
        xx = x[lo]
        j0, j1 = start(xx)
        tp, tc = torch.zeros_like(xx), torch.full_like(xx, 1e-300)
        scale = torch.zeros_like(xx)  # rescalings so far, in units of 1e-200
        kept = {}
        for l in range(L + 31 + int(math.sqrt(40.0 * (L + 2))), 0, -1):
            tm = (2 * l + 1) / xx * tc - tp
            if l in pos:
                kept[l] = (tc, (l * tm - (l + 1) * tp) / (2 * l + 1), scale)
            tp, tc = tc, tm
            big = tc.abs() > 1e200
            f = torch.where(big, torch.full_like(xx, 1e-200), torch.ones_like(xx))
            tp, tc, scale = tp * f, tc * f, scale + big
        if 0 in pos:
            kept[0] = (tc, -tp, scale)
        norm = torch.where(j0.abs() >= j1.abs(), j0 / tc, j1 / tp)
        for l, (v, d, s) in kept.items():
            f = norm * torch.pow(torch.full_like(xx, 1e-200), scale - s)
            y[pos[l], lo], dy[pos[l], lo] = v * f, d * f
    if 0 in pos:
        y[pos[0], 0] = 1.0
    if 1 in pos:
        dy[pos[1], 0] = 1.0 / 3.0
    y[:, N], dy[:, N] = y[:, N - 1], dy[:, N - 1]
    return y, dy, step, dx


def _interp_rows(x, step, dx, hermite=True):
    """Table rows and Hermite (or linear) weights for arguments x."""
    w = x * (1.0 / step)
    i = w.to(torch.int64)
    w = w - i
    v = w - 1
    if not hermite:
        return i, (1 - w, w, 0 * w, 0 * w)
    return i, ((1 + 2 * w) * v * v, w * w * (3 - 2 * w), w * v * v * dx, w * w * v * dx)


def _los(src, ls, taus, ks, xmax):
    """Theta [nk][nl][nsrc] of sources [ntau][nk][nsrc] (trapezoid in tau)."""
    y, dy, step, dx = _bessel_rows(ls, xmax)
    dev = y.device
    src = torch.as_tensor(src, dtype=torch.float64, device=dev)
    k = torch.as_tensor(ks, dtype=torch.float64, device=dev)
    w = np.zeros(len(taus))
    w[:-1] += 0.5 * np.diff(taus)
    w[1:] += 0.5 * np.diff(taus)
    out = torch.zeros((len(ls), len(ks), src.shape[2]), dtype=torch.float64, device=dev)
    for t in range(len(taus)):
        i, c = _interp_rows(k * float(taus[-1] - taus[t]), step, dx)
        j = c[0] * y[:, i] + c[1] * y[:, i + 1] + c[2] * dy[:, i] + c[3] * dy[:, i + 1]
        for s in range(src.shape[2]):
            out[:, :, s] += j * (float(w[t]) * src[t, :, s])
    return out.permute(1, 0, 2).cpu().numpy()


def _spline_m(x, Y):
    """Second derivatives of the natural cubic splines through (x, Y[:, j])."""
    n = len(x)
    h = np.diff(x)
    d = 6 * np.diff(np.diff(Y, axis=0) / h[:, None], axis=0)
    z = np.zeros_like(Y)
    c, e = np.zeros(n), np.zeros_like(Y)
    for i in range(1, n - 1):
        den = 2 * (h[i - 1] + h[i]) - h[i - 1] * c[i - 1]
        c[i] = h[i] / den
        e[i] = (d[i - 1] - h[i - 1] * e[i - 1]) / den
    for i in range(n - 2, 0, -1):
        z[i] = e[i] - c[i] * z[i + 1]
    return z


def _spline_at(x, Y, xq):
    z = _spline_m(x, Y)
    i = np.clip(np.searchsorted(x, xq, side="right") - 1, 0, len(x) - 2)
    h = (x[i + 1] - x[i])[:, None]
    a, b = x[i + 1][:, None] - xq[:, None], xq[:, None] - x[i][:, None]
    return z[i] * a**3 / (6 * h) + z[i + 1] * b**3 / (6 * h) + (Y[i + 1] / h - z[i + 1] * h / 6) * b + (Y[i] / h - z[i] * h / 6) * a


def _kint(A, B, P0, ks):
    """Integral over k of 2/pi k^2 P0 A B through natural splines with the point (0, 0)."""
    x = np.concatenate([[0.0], ks])
    Y = np.concatenate([np.zeros((1, A.shape[1])), (2 / np.pi * ks**2 * P0)[:, None] * A * B])
    z = _spline_m(x, Y)
    h = np.diff(x)[:, None]
    return np.sum(0.5 * h * (Y[1:] + Y[:-1]) - h**3 * (z[1:] + z[:-1]) / 24, axis=0)


def _mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _layers(p, sizes, dev):
    out, o = [], 0
    for a, b in zip(sizes[:-1], sizes[1:]):
        out.append(torch.tensor(p[o:o + a * b].reshape(b, a), dtype=torch.float64, device=dev))
        out.append(torch.tensor(p[o + a * b:o + a * b + b], dtype=torch.float64, device=dev))
        o += a * b + b
    return out


def _forward(L, x):
    for i in range(0, len(L), 2):
        x = x @ L[i].T + L[i + 1]
        if i + 2 < len(L):
            x = x * torch.sigmoid(x)
    return x


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("pk", "factors", "cmb"):
        return None  # a stiff integration of the Boltzmann hierarchy for every mode
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "cmb_sources":
        p = _pars(rng, False)
        t0 = _tau0(p)
        ks = np.geomspace(case["kmin"], case["kmax"], case["nk"]) * HMPC
        taus = 0.01 + (t0 - 0.01) * (1 - np.cos(np.pi * np.linspace(0, 0.5, case["ntau"])))
        ls = _ls(case)
        src = _line_sources(rng, ks, taus, 3)[:, :, :2]
        kf = np.linspace(ks[0], ks[-1], int(math.ceil((ks[-1] - ks[0]) / (np.pi / t0))) + 1)
        fine = _spline_at(np.log(ks), src.reshape(len(ks), -1), np.log(kf)).reshape(len(kf), len(taus), 2).transpose(1, 0, 2).copy()
        fine[-1] = 0
        Th = _los(fine, ls, taus, kf, 20.0 * int(ls[-1]))
        l = ls.astype(np.float64)
        Th[:, :, 0] /= kf[:, None]
        Th[:, :, 1] *= np.sqrt((l + 2) * (l + 1) * l * (l - 1))[None, :] / kf[:, None] ** 2
        kp = 0.05 * HMPC / p["h"]
        P0 = 2 * np.pi**2 * math.exp(p["ln_As1e10"]) / 1e10 / kf**3 * (kf / kp) ** (p["ns"] - 1)
        col = {"T": 0, "E": 1}
        D = np.stack([_kint(Th[:, :, col[m[0]]], Th[:, :, col[m[1]]], P0, kf) for m in case["modes"].split(" ")], axis=1)
        D *= (l * (l + 1) / (2 * np.pi))[:, None]
        return {"Dl": _spline_at(l, D, np.arange(2, int(ls[-1]) + 1).astype(np.float64))}
    if kind == "los":
        t0 = 3.2
        ks = np.linspace(case["kmax"] / case["nk"], case["kmax"], case["nk"])
        taus = 0.01 + (t0 - 0.01) * (1 - np.cos(np.pi * np.linspace(0, 0.5, case["ntau"])))
        ls = _ls(case)
        src = _line_sources(rng, ks, taus, case["nsrc"]).transpose(1, 0, 2)
        P0 = 2 * np.pi**2 * 2.1e-9 / ks**3 * (ks / 100.0) ** (-0.035)
        Th = _los(src.copy(), ls, taus, ks, max(20.0 * int(ls[-1]), 1.01 * t0 * case["kmax"]))
        return {"Theta": Th, "Cl": _kint(Th[:, :, 0], Th[:, :, -1], P0, ks)}
    if kind == "bessel":
        ls = _ls(case)
        xmax = 20.0 * int(ls[-1])
        xs = torch.tensor(rng.uniform(0.0, xmax, case["nx"]), device=dev)
        y, dy, step, dx = _bessel_rows(ls, xmax)
        i, c = _interp_rows(xs, step, dx, case["hermite"])
        at = sorted({0, len(ls) // 3, len(ls) // 2, len(ls) - 1})
        return {"j": np.stack([(c[0] * y[q, i] + c[1] * y[q, i + 1] + c[2] * dy[q, i] + c[3] * dy[q, i + 1]).cpu().numpy() for q in at])}
    sizes, p = _net_params(case, rng)
    X, Y = _net_data(case, rng)
    L = _layers(p, sizes, dev)
    if kind == "mlp_infer":
        X = torch.tensor(X, device=dev)
        return {"Y": torch.cat([_forward(L, X[i:i + 16384].double()) for i in range(0, len(X), 16384)]).cpu().numpy()}
    # training: Adam (0.9, 0.999, 1e-8) on the network's own uniform batches (seed 1)
    X, Y = torch.tensor(X, device=dev), torch.tensor(Y, device=dev)
    m, v = [torch.zeros_like(q) for q in L], [torch.zeros_like(q) for q in L]
    i = np.arange(case["batch"], dtype=np.uint64)
    loss = 0.0
    for t in range(1, case["steps"] + 1):
        with np.errstate(over="ignore"):
            r = _mix64(np.uint64(1) ^ _mix64(np.uint64(t) * np.uint64(0x100000001B3) + i)) % np.uint64(case["rows"])
        r = torch.tensor(r.astype(np.int64), device=dev)
        g = [torch.zeros_like(q) for q in L]
        loss = 0.0
        for o in range(0, case["batch"], 16384):
            leaf = [q.clone().requires_grad_(True) for q in L]
            b = r[o:o + 16384]
            e = ((_forward(leaf, X[b].double()) - Y[b].double()) ** 2).sum() / (case["batch"] * case["nout"])
            for q, d in zip(g, torch.autograd.grad(e, leaf)):
                q += d
            loss += float(e)
        for j in range(len(L)):
            m[j] = 0.9 * m[j] + 0.1 * g[j]
            v[j] = 0.999 * v[j] + 0.001 * g[j] ** 2
            L[j] = L[j] - 2e-4 * (m[j] / (1 - 0.9**t)) / (torch.sqrt(v[j] / (1 - 0.999**t)) + 1e-8)
    return {"loss": loss, "params": np.concatenate([q.cpu().numpy().ravel() for q in L])}
