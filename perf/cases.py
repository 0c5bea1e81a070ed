"""Performance cases of the opacity path: the calls a user's program makes.

Every case builds a synthetic line list or spectrum from its seed on the GPU,
hands it to the framework as such a program would (``prepare``), and makes one
pass through the public entry points (``run``).  ``exact`` restates the same
result in 64-bit torch.  Line distributions are those of hkb.synth; grids,
cutoffs, states and orders are those of the repository's workloads and tests,
with odd sizes beside the round ones.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "helios-k_b200"))
import hkb  # noqa: E402
from hkb import synth  # noqa: E402
from hkb.autograd import Opacity  # noqa: E402

E_MAX = 25000.0  # largest lower-state energy, cm-1
LINES = dict(database="hitran", numin=0.0, dnu=0.01, cut=25.0, nbins=1, precision="mixed",
             logS0=-30.0, logS1=-18.0, E=3000.0, shift=False, plinth=False,
             T0=1000.0, T1=1000.0, nT=1, P0=1.0, P1=1.0, nP=1, nC=20)


def listed():
    """Twelve cases, the smallest call first."""
    c = []

    def lines(name, **kw):
        c.append(dict(LINES, name=name, **kw))

    # one band of one molecule at room temperature, K on the device: the
    # smallest call, made once per layer by a line-by-line radiative transfer
    lines("band", kind="opacity", n=2000, numin=1000.0, nx=10000, T0=296.0, T1=296.0)
    # a ragged band with pressure shifts and Einstein coefficients (HITRAN
    # columns that vary), K and the fit returned to host memory
    lines("band_host", kind="fit", n=12347, numin=667.1, nx=33333, dnu=0.003, nbins=3, shift=True,
          host=True, T0=250.0, T1=250.0, P0=0.1, P1=0.1)
    # 1e5 lines on the full grid, cut 100 cm-1, K and its k-distribution fit
    lines("state", kind="fit", n=100_000, nx=3_000_000, cut=100.0, nbins=300)
    # 1e7 lines (HITEMP size) on the full grid: the flagship state
    lines("state_dense", kind="fit", n=10_000_000, nx=3_000_000, nbins=300, logS0=-32.0,
          T0=1500.0, T1=1500.0, P0=0.1, P1=0.1)
    # a T-P table with uneven windows, one graph replay
    lines("table", kind="table", n=300_000, nx=300_000, nbins=30, logS0=-32.0, T0=100.0, T1=3000.0,
          nT=4, P0=1e-8, P1=1e3, nP=6)
    # an ExoMol list (fixed widths), a batch of states, K only
    lines("exomol", kind="opacity", database="exomol", n=2_500_000, nx=1_000_000, logS0=-40.0,
          E=8000.0, T0=500.0, T1=2500.0, nT=2, P0=1e-4, P1=10.0, nP=2)
    # the plain FP64 form, which a user takes to check the mixed one
    lines("plain", kind="opacity", n=60_000, nx=300_000, precision="plain")
    # water with a continuum: the plinth at the 25 cm-1 cut is removed
    lines("plinth", kind="opacity", n=100_000, numin=500.0, nx=200_000, plinth=True, T0=400.0,
          T1=400.0, P0=0.3, P1=0.3)
    # refit of stored spectra: sort, Chebyshev fit and reconstruction
    c.append(dict(name="refit", kind="refit", states=16, nx=300_000, nbins=30, nC=20))
    # Planck / Rosseland means and transmission functions of stored spectra
    c.append(dict(name="means", kind="means", states=6, nx=300_000, nbins=30, nTr=1000, dTr=0.05,
                  T0=400.0, T1=2400.0))
    # one step of a retrieval: K of a band, loss on log K, gradients of T, P
    # and every line's strength and width
    lines("retrieval", kind="gradient", n=30_000, numin=2000.0, nx=50_000, T0=800.0, T1=800.0)
    # the same step at the size of the gradient workload
    lines("retrieval_wide", kind="gradient", n=1_000_000, numin=1000.0, nx=900_000, cut=100.0,
          T0=800.0, T1=800.0)
    return c


def draw(rng):
    """One more case of the same kinds and ranges."""
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["opacity", "opacity", "fit", "fit", "table", "gradient", "refit", "means"])
    nbins = rng.randint(1, 40)
    nxb = int(log(1500, 11000))
    if kind == "refit":
        return dict(kind=kind, states=rng.randint(1, 16), nx=nbins * nxb, nbins=nbins,
                    nC=rng.randint(8, 30))
    if kind == "means":
        return dict(kind=kind, states=rng.randint(1, 6), nx=nbins * nxb, nbins=nbins,
                    nTr=rng.randint(200, 1100), dTr=0.05, T0=rng.uniform(150.0, 800.0),
                    T1=rng.uniform(900.0, 2900.0))
    dnu = rng.choice([0.01, 0.01, 0.005, 0.02, 0.0137])
    c = dict(LINES, kind=kind, nbins=nbins, nx=nbins * nxb, dnu=dnu,
             cut=rng.choice([25.0, 25.0, 50.0, 100.0]),
             numin=rng.choice([0.0, round(rng.uniform(100.0, 6000.0), 1)]))
    span = c["nx"] * dnu
    # 10 to 300 lines per wavenumber
    c["n"] = max(400, min(1_000_000, int(log(10.0, 300.0) * span)))
    T, P = rng.uniform(150.0, 2900.0), log(1e-4, 10.0)
    c.update(T0=T, T1=T, P0=P, P1=P)
    if kind == "opacity":
        opt = rng.choice(["exomol", "exomol", "mixed", "mixed", "plain", "plinth"])
        if opt == "exomol":
            c.update(database="exomol", logS0=-40.0, E=8000.0, T1=min(2900.0, 1.5 * T), nT=2)
        elif opt == "plain":
            c.update(precision="plain", n=min(c["n"], 60_000), cut=25.0)
        elif opt == "plinth":
            c.update(plinth=True, n=min(c["n"], 100_000), cut=25.0)
    elif kind == "fit":
        c.update(shift=rng.random() < 0.5, host=rng.random() < 0.3, nC=rng.randint(8, 30))
    elif kind == "table":
        c.update(n=min(c["n"], 300_000), T0=rng.uniform(100.0, 400.0), T1=3000.0,
                 nT=rng.randint(2, 4), P0=1e-8, P1=1e3, nP=rng.randint(2, 6), logS0=-32.0)
    return c


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, a, b):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (b - a) + a


def _numax(c):
    return c["numin"] + c["nx"] * c["dnu"]


def _lines(c, seed):
    """Line columns (CUDA float64) with the distributions of hkb.synth, drawn
    over the grid and a cutoff's reach beyond it."""
    g = _generator(seed)
    n = c["n"]
    lo = max(1e-3, c["numin"] - c["cut"])
    hi = _numax(c) + (c["cut"] if c["numin"] > 0.0 else 0.0)
    f = float(synth.q_of_T(296.0)) / (synth.MASS / synth.NA)
    L = dict(nu=_uniform(g, n, lo, hi),
             S=torch.pow(10.0, _uniform(g, n, c["logS0"], c["logS1"])) * f,
             # lower-state energies end where real lists do (dissociation)
             EL=-torch.log1p(-_uniform(g, n, 0.0, 1.0 - math.exp(-E_MAX / c["E"]))) * c["E"])
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    L["A"] = zero
    if c["database"] == "hitran":
        L["gair"] = _uniform(g, n, 0.01, 0.1)
        L["gself"] = L["gair"]
        L["n"] = _uniform(g, n, 0.4, 0.8)
        L["delta"] = zero
        if c["shift"]:
            L["gself"] = _uniform(g, n, 0.01, 0.5)
            L["delta"] = _uniform(g, n, -0.01, 0.01)
            L["A"] = torch.pow(10.0, _uniform(g, n, -6.0, 1.5))
    return L


def _states(c):
    T = np.linspace(c["T0"], c["T1"], c["nT"])
    P = np.exp(np.linspace(math.log(c["P0"]), math.log(c["P1"]), c["nP"]))
    TT, PP = np.meshgrid(T, P, indexing="ij")
    return TT.ravel(), PP.ravel()


def _spectra(c, seed):
    """Stored opacities (states, nx) in cm2/g: lines of 12 decades of strength
    with Lorentz wings over a continuum floor."""
    g = _generator(seed)
    ns, nx = c["states"], c["nx"]
    spikes = torch.zeros(ns, nx, dtype=torch.float64, device="cuda")
    m = max(8, nx // 60)
    at = torch.randint(0, nx, (ns, m), generator=g, device="cuda")
    s = torch.pow(10.0, _uniform(g, ns * m, -7.0, 5.0)).view(ns, m)
    spikes.scatter_add_(1, at, s)
    k = torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) * (2.0 * math.pi / nx)
    width = torch.linspace(0.5, 12.0, ns, device="cuda", dtype=torch.float64).view(ns, 1)
    K = torch.fft.irfft(torch.fft.rfft(spikes) * torch.exp(-k * width), n=nx)
    return K.clamp_min(0.0) + _uniform(g, ns * nx, 0.5e-8, 2e-8).view(ns, nx)


def _context(c, seed):
    ctx = hkb.Context(torch.cuda.current_device())
    Tq, Qq = synth.q_table()
    L = {k: v.cpu().numpy() for k, v in _lines(c, seed).items()}
    if c["database"] == "exomol":
        ctx.set_species(hkb.EXOMOL, [synth.MASS], [1.0], 0.07, 0.5)
        ctx.set_partition(0, Tq, Qq)
        ctx.load_lines_exomol(L)
    else:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=0.5)
        ctx.load_lines_hitran(L)
    ctx.set_grid(c["numin"], _numax(c), c["dnu"], c["nbins"], 0, c["cut"])
    if ctx.nx != c["nx"]:
        raise ValueError("the grid holds %d points, not %d" % (ctx.nx, c["nx"]))
    if c["plinth"]:
        ctx.set_profile(1, 1)
    return ctx


def _retrieval_inputs(c, seed):
    g = _generator(seed + 1_000_003)
    n = c["n"]
    w = torch.randn(c["nx"], generator=g, device="cuda", dtype=torch.float64)
    log_s = 0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    log_g = 0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return w, log_s, log_g


class State:
    pass


def prepare(case, seed):
    c, s = case, State()
    s.case = c
    if c["kind"] in ("refit", "means"):
        s.K = _spectra(c, seed)
        s.ctx = hkb.Context(torch.cuda.current_device())
        s.ctx.set_grid(0.0, c["nx"] * 0.01, 0.01, c["nbins"], 0, 25.0)
        if c["kind"] == "means":
            s.T = np.linspace(c["T0"], c["T1"], c["states"])
            s.fit = s.ctx.kdist(s.K, nC=20, recon=True)
        return s
    s.ctx = _context(c, seed)
    s.T, s.P = _states(c)
    ns = len(s.T)
    s.precision = hkb.PLAIN_FP64 if c["precision"] == "plain" else hkb.MIXED
    if c["kind"] == "gradient":
        s.w, log_s, log_g = _retrieval_inputs(c, seed)
        s.leaves = [torch.tensor(c["T0"], dtype=torch.float64, requires_grad=True),
                    torch.tensor(c["P0"], dtype=torch.float64, requires_grad=True),
                    log_s.requires_grad_(), log_g.requires_grad_()]
    elif not c.get("host", False):
        s.K = torch.empty(ns, c["nx"], dtype=torch.float64, device="cuda")
    if c["kind"] == "table":
        s.coeff = torch.empty(ns, c["nbins"], c["nC"], dtype=torch.float64, device="cuda")
        s.nxmin = torch.empty(ns, c["nbins"], dtype=torch.int32, device="cuda")
        s.ctx.table_build(s.T, s.P, s.K, s.coeff, s.nxmin, nC=c["nC"])
    return s


def run(s):
    c, ctx = s.case, s.ctx
    kind = c["kind"]
    if kind == "refit":
        r = ctx.kdist(s.K, nC=c["nC"], sorted_K=True, recon=True)
        return [r["coeff"], r["sorted"], r["recon"], r["nxmin"]]
    if kind == "means":
        sums = ctx.means(s.T, s.K)
        tr = ctx.transmission(s.fit["recon"], s.fit["nxmin"], nTr=c["nTr"], dTr=c["dTr"])
        return [sums, tr]
    if kind == "table":
        ctx.table_run()
        return [s.K, s.coeff, s.nxmin]
    if kind == "gradient":
        K = Opacity.apply(ctx, *s.leaves)
        loss = torch.dot(s.w, torch.log(K))
        return list(torch.autograd.grad(loss, s.leaves)) + [loss.detach()]
    K = ctx.opacity(s.T, s.P, s.precision, out=None if c.get("host", False) else s.K)
    if kind == "opacity":
        return [K]
    r = ctx.kdist(K, nC=c["nC"])
    return [K, r["coeff"], r["nxmin"]]


def work(case):
    """Inputs read once, outputs written once; a line evaluation of 8 flops (a
    Lorentzian and its sum) per grid point inside a line's window, 12 for the
    derivatives, and the fit's, the means' and the transmission's sums."""
    c = case
    kind = c["kind"]
    if kind in ("refit", "means"):
        K = 8.0 * c["states"] * c["nx"]
        if kind == "refit":
            return {"bytes": 3.0 * K, "flops": K / 8.0 * (4.0 * c["nC"] + 40.0)}
        return {"bytes": 2.0 * K + 8.0 * c["states"] * c["nbins"] * c["nTr"],
                "flops": K / 8.0 * (20.0 * c["nTr"] + 60.0)}
    ns = c["nT"] * c["nP"]
    cols = 3 if c["database"] == "exomol" else (7 if c["shift"] else 5)
    span = c["nx"] * c["dnu"]
    reach = span + (2.0 if c["numin"] > 0.0 else 1.0) * c["cut"]
    pairs = ns * c["n"] * min(c["nx"], 2.0 * c["cut"] / c["dnu"]) * min(1.0, span / reach)
    b = 8.0 * cols * c["n"] + 8.0 * ns * c["nx"]
    f = 8.0 * pairs
    if kind == "gradient":
        b += 8.0 * (c["nx"] + 4.0 * c["n"])
        f += 12.0 * pairs
    elif kind != "opacity":
        b += 8.0 * ns * c["nx"]
        f += ns * c["nx"] * (2.0 * c["nC"] + 40.0)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- 64-bit restatement

PI = math.pi
HC_K = 6.62606957e-27 * 2.99792458e10 / 1.3806489e-16
NA = 6.0221412927e23


def _partition(T):
    """Q(T) of the 1 K table, linear inside the segment below T."""
    t0 = math.ceil(float(T.detach())) - 1.0
    q0, q1 = float(synth.q_of_T(t0)), float(synth.q_of_T(t0 + 1.0))
    return q0 + (q1 - q0) * (T - t0)


def _scaled(c, L, T, P, log_s=None, log_g=None):
    """Line centre, strength times 1/alphaD, 1/alphaD and gammaL/alphaD."""
    iad0 = 2.99792458e10 * torch.sqrt(synth.MASS / NA / (2.0 * 1.3806489e-16 * T))
    if c["database"] == "exomol":
        nu = L["nu"]
        S = L["S"] / _partition(T) * torch.exp(-HC_K / T * L["EL"]) * (1.0 - torch.exp(-HC_K / T * nu))
        aL = 0.07 * (P / 0.986923) * torch.sqrt(296.0 / T) + L["A"] / (4.0 * PI * 2.99792458e10)
    else:
        nu = L["nu"] + L["delta"] * P
        S = L["S"] / _partition(T) * torch.exp(HC_K * L["EL"] * (1.0 / 296.0 - 1.0 / T)) * \
            (1.0 - torch.exp(-HC_K * nu / T)) / (1.0 - torch.exp(-HC_K * nu / 296.0))
        gam = 0.5 * L["gair"] + 0.5 * L["gself"]
        aL = gam * P * torch.pow(296.0 / T, L["n"]) + L["A"] / (4.0 * PI * 2.99792458e10)
    if log_s is not None:
        S, aL = S * torch.exp(log_s), aL * torch.exp(log_g)
    iad = iad0 / nu
    return nu, S * iad, iad, aL * iad


def _voigt(x, y):
    """Re w(x + iy) for r < 10 by the exponentially convergent trapezoidal
    series (Zaghloul & Ali 2011), step 1/2."""
    a = 0.5
    x = x.abs()
    ex, c2, sn = torch.exp(-x * x), torch.cos(2.0 * x * y), torch.sin(x * y)
    t = torch.zeros_like(x)
    for n in range(1, 35):
        an = a * n
        g = 0.5 * torch.exp(-(an - x) ** 2)
        if n < 14:
            g = g + 0.5 * torch.exp(-(an + x) ** 2) - c2 * ex * math.exp(-an * an)
        t = t + g / (an * an + y * y)
    return ex * torch.special.erfcx(y) * c2 + (2.0 * a / PI) * (ex * sn * sn / y + y * t)


def _gh2(s, Y):
    u = s + Y
    return ((u + 1.5) * (u + 1.0) - (4.0 / PI) * s) / (u * ((u + 1.5) ** 2 - (6.0 / PI) * s))


def _chunks(c, nu, iad, y, Sx):
    """Per chunk of lines: (line index, grid index, x, y, S/alphaD, region C)
    of the points inside the cut window, regions C and A/B apart."""
    W = min(c["nx"], int(2.0 * c["cut"] / c["dnu"]) + 3)
    per = max(1, (1 << 23) // W)
    off = torch.arange(W, device="cuda")
    for l0 in range(0, len(nu), per):
        sl = slice(l0, min(len(nu), l0 + per))
        v = nu[sl].detach()
        first = torch.ceil((v - c["cut"] - c["numin"]) / c["dnu"]).long() - 1
        first = first.clamp(0, c["nx"] - W)
        idx = first[:, None] + off
        xg = c["numin"] + idx.double() * c["dnu"]
        inside = (xg - v[:, None]).abs() < c["cut"]
        r2 = ((xg - v[:, None]) * iad[sl].detach()[:, None]) ** 2 + (y[sl].detach() ** 2)[:, None]
        for inC in (True, False):
            li, p = torch.nonzero(inside & ((r2 < 100.0) == inC), as_tuple=True)
            if len(li):
                k = idx[li, p]
                li = li + l0
                x = (c["numin"] + k.double() * c["dnu"] - nu[li]) * iad[li]
                yield li, k, x, y[li], Sx[li], inC


def _term(x, y, Sx, inC):
    if inC:
        return Sx / math.sqrt(PI) * _voigt(x, y)
    s, Y = x * x, y * y
    return Sx * y / PI * torch.where(s + Y < 1e6, _gh2(s, Y), 1.0 / (s + Y))


def _edge(c, nu, iad, y, Sx):
    """Each line's profile at its cut edge."""
    x = c["cut"] * iad
    inC = x * x + y * y < 100.0
    return torch.where(inC, _term(torch.where(inC, x, torch.ones_like(x)), y, Sx, True),
                       _term(x, y, Sx, False))


def _opacity(c, L, T, P, log_s=None, log_g=None):
    T, P = (torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in (T, P))
    with torch.no_grad():
        nu, Sx, iad, y = _scaled(c, L, T, P, log_s, log_g)
        edge = _edge(c, nu, iad, y, Sx) if c["plinth"] else None
        K = torch.zeros(c["nx"], dtype=torch.float64, device="cuda")
        for li, k, x, yy, ss, inC in _chunks(c, nu, iad, y, Sx):
            t = _term(x, yy, ss, inC)
            K.index_add_(0, k, t - edge[li] if c["plinth"] else t)
    return K


def _fit(K, nbins, nC):
    """(sorted, coefficients) of spectra (ns, nx) without empty points: the
    Householder least squares with the first nC - 1 reflections applied."""
    ns, nx = K.shape
    nxb = nx // nbins
    srt = torch.sort(K.view(ns * nbins, nxb), dim=1).values
    x = torch.arange(nxb, dtype=torch.float64) * 2.0 / (nxb - 1.0) - 1.0
    V = torch.cos(torch.acos(x.clamp(-1.0, 1.0))[:, None] * torch.arange(nC, dtype=torch.float64))
    V = V.to(K.device)
    b = torch.log(srt).T.contiguous()
    for j in range(nC):
        v = V[:, j].clone()
        v[:j] = 0.0
        sigma = torch.linalg.norm(v) * (-1.0 if v[j] < 0 else 1.0)
        v[j] += sigma
        h = v / (sigma * v[j])
        V = V - torch.outer(h, v @ V)
        if j < nC - 1:
            b = b - torch.outer(h, v @ b)
    co = torch.linalg.solve_triangular(V[:nC].triu(), b[:nC], upper=True)
    return srt.view(ns, nx), co.T.reshape(ns, nbins, nC).contiguous()


def _recon(co, nxb):
    ns, nbins, nC = co.shape
    x = -1.0 + torch.arange(nxb, dtype=torch.float64, device=co.device) * 2.0 / nxb
    T = torch.cos(torch.acos(x)[:, None] * torch.arange(nC, dtype=torch.float64, device=co.device))
    return torch.exp(torch.einsum("sbj,kj->sbk", co, T)).reshape(ns, nbins * nxb)


def _end_weights(v):
    """Plain sum along the last axis with the end corrections of the sums."""
    w = (-5.0 / 8.0, 1.0 / 6.0, -1.0 / 24.0)
    t = v.sum(-1)
    for k in range(3):
        t = t + w[k] * v[..., k] + w[2 - k] * v[..., -1 - k]
    return t


def _means_exact(c, seed):
    K = _spectra(c, seed)
    ns, nx = K.shape
    nb = c["nbins"]
    nxb = nx // nb
    T = torch.linspace(c["T0"], c["T1"], ns, dtype=torch.float64, device="cuda").view(ns, 1)
    nu = torch.arange(nx, dtype=torch.float64, device="cuda") * 0.01
    h, cl, kB = 6.62606957e-27, 2.99792458e10, 1.3806489e-16
    t1 = 2.0 * h * nu ** 3 * cl * cl
    t2 = h * nu * cl / (kB * T)
    B = torch.where(nu > 0.0, t1 / torch.expm1(t2), torch.zeros_like(t2))
    R = torch.where(nu > 0.0, t1 * t2 / (T * 4.0 * torch.sinh(0.5 * t2) ** 2), torch.zeros_like(t2))
    sums = torch.stack([_end_weights(v) for v in (B * K, R / K, B, R)], dim=1)
    rec = _recon(_fit(K, nb, 20)[1], nxb).view(ns, nb, nxb)
    tr = torch.empty(ns, nb, c["nTr"], dtype=torch.float64, device="cuda")
    for j in range(c["nTr"]):
        tr[:, :, j] = _end_weights(torch.exp(-rec * math.exp((j - c["nTr"] // 2) * c["dTr"]))) / (nxb - 1)
    return [sums, tr]


def _gradient_exact(c, seed):
    L = _lines(c, seed)
    w, log_s, log_g = _retrieval_inputs(c, seed)
    K = _opacity(c, L, c["T0"], c["P0"], log_s, log_g)
    u = w / K
    # dLoss per line in (nu, S/alphaD, 1/alphaD, y), then the line scaling
    with torch.no_grad():
        lin = _scaled(c, L, torch.tensor(c["T0"], dtype=torch.float64, device="cuda"),
                      torch.tensor(c["P0"], dtype=torch.float64, device="cuda"), log_s, log_g)
    lin = [v.clone().requires_grad_() for v in lin]
    got = [torch.zeros_like(v) for v in lin]
    for li, k, x, yy, ss, inC in _chunks(c, lin[0], lin[2], lin[3], lin[1]):
        part = (u[k] * _term(x, yy, ss, inC)).sum()
        for a, b in zip(got, torch.autograd.grad(part, lin, allow_unused=True)):
            if b is not None:
                a += b
    T = torch.tensor(c["T0"], dtype=torch.float64, device="cuda", requires_grad=True)
    P = torch.tensor(c["P0"], dtype=torch.float64, device="cuda", requires_grad=True)
    log_s.requires_grad_()
    log_g.requires_grad_()
    grads = torch.autograd.grad(_scaled(c, L, T, P, log_s, log_g), [T, P, log_s, log_g], got)
    # at a node of the partition table the library takes the mean of the two
    # neighbouring slopes: the slope of ln Q enters every line's strength
    if float(c["T0"]).is_integer():
        t = float(c["T0"])
        q = [float(synth.q_of_T(t + d)) for d in (-1.0, 0.0, 1.0)]
        below, mean = (q[1] - q[0]) / q[1], 0.5 * (q[2] - q[0]) / q[1]
        grads = (grads[0] - (mean - below) * grads[2].sum(),) + tuple(grads[1:])
    return list(grads) + [torch.dot(w, torch.log(K))]


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "means":
        return _means_exact(c, seed)
    if kind == "refit":
        srt, co = _fit(_spectra(c, seed), c["nbins"], c["nC"])
        return [co, srt, _recon(co, c["nx"] // c["nbins"]), None]
    ns = c["nT"] * c["nP"]
    pairs = ns * c["n"] * min(c["nx"], 2.0 * c["cut"] / c["dnu"])
    if pairs > (1e9 if kind == "gradient" else 4e10):
        return None
    if kind == "gradient":
        return _gradient_exact(c, seed)
    L = _lines(c, seed)
    K = torch.stack([_opacity(c, L, T, P) for T, P in zip(*_states(c))])
    if kind == "opacity":
        return [K]
    if not bool((K > 0.0).all()):
        return [K, None, None]
    return [K, _fit(K, c["nbins"], c["nC"])[1], None]
