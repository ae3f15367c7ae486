"""The work a user of the package has it do, as cases that can be timed.

A case is one pass through the package's public entry points on inputs that
are on the GPU already: particles from a parameter set (one realisation, on an
array of Lagrangian positions or on the lattice glass; several as a batch;
streamed over slabs), the non-Gaussian potential of a given Gaussian one, the
displacement field with its gradients, the 3-D transforms, and the mode
covariance and projections of the Decomposer.  `exact` restates each in 64
bits with torch and numpy alone.
"""
import math
import os

import numpy as np
import torch

from aarambam_gb300 import tables
from aarambam_gb300.adjoint import displacement
from aarambam_gb300.basis import Basis
from aarambam_gb300.ic import ICBatch, ICGenerator

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = torch.device("cuda")
F64 = torch.float64

# Cosmology and units of the parameter files (z = 49, BBKS transfer function).
BASE = dict(Omega=0.3, OmegaLambda=0.7, OmegaBaryon=0.0, OmegaDM_2ndSpecies=0.0, HubbleParam=0.7, ShapeGamma=0.0,
            Sigma8=0.8, PrimordialIndex=0.965, Redshift=49.0, FixedAmplitude=0, PhaseFlip=0, SavePotentialField=0,
            WhichSpectrum=0, WhichTransfer=2, InputSpectrum_UnitLength_in_cm=3.085678e24,
            UnitLength_in_cm=3.085678e24, UnitMass_in_g=1.989e43, UnitVelocity_in_cm_per_s=1e5)

# Templates: coefficient table (None: the few exact coefficients below), modes,
# box (Mpc/h) and the largest Nmesh the table was made for.  Local and
# Equilateral are exact sums of the first modes, so they serve any box.
TEMPLATES = {
    "local6": (None, 6, 500.0, 1024), "local8": (None, 8, 500.0, 1024), "equil9": (None, 9, 500.0, 1024),
    "scalarI10": ("scalarI_m10_L500_n256", 10, 500.0, 256),
    "scalarI12": ("scalarI_m12_L1000_n512", 12, 1000.0, 512),
    "scalarI13": ("scalarI_m13_L500_n256_mu0p5", 13, 500.0, 256),
    "scalarI16": ("scalarI_m16_L500_n256_mu1p5", 16, 500.0, 256),
    "scalarI20": ("scalarI_m20_L500_n256_mu1p75", 20, 500.0, 256),
}
EXACT_TERMS = {"local": [(0, 0, 3, 1.0)], "equil": [(0, 0, 3, -3.0), (0, 1, 2, 6.0), (1, 1, 1, -2.0)]}
BATCH = ["local6", "equil9", "scalarI10", "scalarI13", "scalarI16", "scalarI20"]


def listed():
    return [
        # the smallest whole call: quick looks, tests, many small boxes; a glass-like load, odd particle count
        dict(name="run_64", kind="run", N=64, template="scalarI10", particles=250047, sphere=0),
        # one realisation as the plain parameter file has it: 128^3, Local, a lattice of particles as an array
        dict(name="run_128_local", kind="run", N=128, template="local8", particles=128 ** 3, sphere=0),
        # production sizes through the lattice glass, ScalarI templates; 512^3 is the precision configuration
        dict(name="lattice_256", kind="lattice", N=256, template="scalarI13", sphere=1),
        dict(name="lattice_512", kind="lattice", N=512, template="scalarI12", sphere=0),
        # the largest grid of the fused form, Local (its 20-mode state would not fit the card several times)
        dict(name="lattice_1024_local", kind="lattice", N=1024, template="local8", sphere=0),
        # realisations with uneven templates in one graph
        dict(name="batch_128", kind="batch", N=128, count=6),
        # the potential of a Gaussian field the caller has (modal split, constrained realisations), most modes
        dict(name="potential_256", kind="potential", N=256, template="scalarI20", sphere=0),
        # inference steps: displacement field and its gradients, small and at the differentiation configuration
        dict(name="gradient_64", kind="gradient", N=64, template="scalarI10"),
        dict(name="gradient_256", kind="gradient", N=256, template="scalarI10"),
        # the transforms a user calls between steps of an own analysis
        dict(name="transforms_512", kind="transforms", N=512, fields=1),
        # one table's covariance and first projection in the Decomposer, 20 modes on the standard grid
        dict(name="covariance_20", kind="covariance", modes=20, grid=150, Nmax=1536),
        # grids streamed over slabs, a factor 3 in N
        dict(name="slab_384", kind="slab", N=384, template="scalarI12", slabs=8),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "lattice", "lattice", "batch", "potential", "gradient", "transforms",
                       "covariance", "slab"])
    names = sorted(TEMPLATES)
    if kind == "covariance":
        return dict(kind=kind, modes=rng.randint(5, 20), grid=rng.randint(40, 150), Nmax=rng.choice([128, 256, 1536]))
    if kind == "transforms":
        return dict(kind=kind, N=rng.choice([32, 64, 128, 256]), fields=rng.randint(2, 6))
    if kind == "batch":
        return dict(kind=kind, N=rng.choice([32, 64, 128]), count=rng.randint(2, 6), first=rng.randint(1, len(BATCH) - 1))
    if kind == "slab":
        N, slabs = rng.choice([(48, 2), (96, 4), (144, 6), (192, 8), (256, 4), (288, 8), (320, 5), (384, 6), (384, 8)])
        case = dict(kind=kind, N=N, slabs=slabs)
    else:
        N = rng.choice({"run": [32, 64, 128, 256, 512], "lattice": [32, 64, 128, 256, 512],
                        "potential": [32, 64, 128, 256], "gradient": [32, 64, 128, 256]}[kind])
        case = dict(kind=kind, N=N, sphere=rng.choice([0, 0, 1]))
    case["template"] = rng.choice([n for n in names if TEMPLATES[n][3] >= N and
                                   (kind != "gradient" or TEMPLATES[n][1] <= 13)])
    # modes above a part of the Nyquist frequency cut, as runs that compare resolutions do
    case["Nsample"] = N if rng.random() < 0.5 else 2 * rng.randint(N // 4, N // 2 - 1)
    if kind == "run":
        case["particles"] = int(N ** 3 * math.exp(rng.uniform(math.log(0.05), 0.0)))
    return case


# ------------------------------------------------------------------ inputs
def _template(name):
    """alpha[M][M][M], X0[M] of a template (X0: the Legendre polynomials at k = 0, as generate_Ai makes them)."""
    tab, M, L, nmax = TEMPLATES[name]
    if tab is None:
        alpha = np.zeros((M, M, M))
        for p, q, r, v in EXACT_TERMS["local" if name.startswith("local") else "equil"]:
            for x, y, z in ((p, q, r), (p, r, q), (q, p, r), (q, r, p), (r, p, q), (r, q, p)):
                alpha[x, y, z] = v
    else:
        alpha = tables.load_alpha(os.path.join(ROOT, "tests", "golden", "tables", tab, "AlphaTable.dat"), M)
    s = (4 - BASE["PrimordialIndex"]) / 3
    a, b = (2 * np.pi / L) ** s, (2 * np.pi / L * nmax) ** s
    at = -1 - 2 * a / (b - a)
    x0 = [1.0, at]
    for l in range(2, M):
        x0.append(((2 * l - 1) * at * x0[-1] - (l - 1) * x0[-2]) / l)
    return alpha, np.array(x0[:M])


def _cfg(case, seed, template=None):
    _, M, L, nmax = TEMPLATES[template or case["template"]]
    return dict(BASE, Nmesh=case["N"], Nsample=case.get("Nsample", case["N"]), Nmax=nmax, Box=L, Seed=int(seed) % 2000000011 + 1,
                Fnl=100.0, N_modes=M, SphereMode=int(case.get("sphere", 0)))


def _rng(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _lattice(N, box):
    g = torch.arange(N, device=DEV, dtype=torch.float32) * np.float32(box / N)
    return torch.stack([x.reshape(-1) for x in torch.meshgrid(g, g, g, indexing="ij")], 1).contiguous()


def _particles(case, seed, box):
    """A lattice where the count is N^3, else that many glass-like positions of a slab of the box, in its order."""
    n, N = case["particles"], case["N"]
    if n == N ** 3:
        return _lattice(N, box)
    m = math.ceil(n ** (1 / 3))
    i = torch.arange(n, device=DEV)
    cell = torch.stack([i // (m * m), (i // m) % m, i % m], 1).to(F64)
    u = torch.rand((n, 3), generator=_rng(seed, 1), device=DEV, dtype=F64)
    return ((cell + u) * (box / m)).to(torch.float32).clamp_(0.0, float(np.nextafter(np.float32(box), np.float32(0))))


def _noise(N, seed):
    """Unit-variance complex noise on the half spectrum, as the path's own draw makes it."""
    g = _rng(seed, 2)
    u = torch.rand((2, N, N, N // 2 + 1), generator=g, device=DEV, dtype=F64)
    return torch.polar(torch.sqrt(-torch.log1p(-u[0])), 2 * math.pi * u[1]).to(torch.complex64)


def _shapes(basis_grid, seed, n=2):
    """Shape functions (k1 k2 k3)^2 B on tetrapyd points: smooth, scale-invariant envelopes with an oscillation."""
    r = np.random.default_rng(int(seed) % (1 << 32))
    k1, k2, k3 = basis_grid
    kt = k1 + k2 + k3
    out = []
    for _ in range(n):
        w, ph = r.uniform(2, 8), r.uniform(0, 2 * np.pi)
        out.append((k1 * k2 * k3) ** 0.01 * (1 + 0.5 * np.cos(w * np.log(kt) + ph)))
    return np.stack(out)


def _grid_case(case, seed):
    """k range of a covariance case: the box varies a little with the seed."""
    L = 2000.0 * (1 + 0.01 * (int(seed) % 97) / 97)
    kF = 2 * np.pi / L
    return kF, kF * case["Nmax"]


def _batch(case):
    return [BATCH[(case.get("first", 0) + i) % len(BATCH)] for i in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "covariance":
        kmin, kmax = _grid_case(case, seed)
        s["basis"] = Basis(kmin, kmax, BASE["PrimordialIndex"], case["modes"], case["grid"], verbose=False)
        s["S"] = _shapes(s["basis"].tetrapyd_grid, seed)
        return s
    k, T = tables.bbks_transfer()
    if kind == "batch":
        gens = []
        for i, t in enumerate(_batch(case)):
            gens.append(ICGenerator(_cfg(case, int(seed) + 7919 * i, t), *_template(t), k, T))
        s["gens"], s["batch"] = gens, ICBatch(gens)
        s["lagr"] = [_lattice(case["N"], g.cfg["Box"]) for g in gens]
        s["pos"] = [torch.empty_like(x) for x in s["lagr"]]
        s["vel"] = [torch.empty_like(x) for x in s["lagr"]]
        return s
    if kind == "transforms":
        cfg = _cfg(dict(case, template="local6"), seed)
        s["gen"] = ICGenerator(cfg, *_template("local6"), k, T)
        s["real"], s["spec"] = _transform_input(case, seed)
        return s
    cfg = _cfg(case, seed)
    alpha, x0 = _template(case["template"])
    form = dict(precision="slab_fp32", nslab=case["slabs"]) if kind == "slab" else {}
    s["gen"] = gen = ICGenerator(cfg, alpha, x0, k, T, **form)
    N, box = case["N"], cfg["Box"]
    if kind == "run":
        s["lagr"] = _particles(case, seed, box)
        s["pos"], s["vel"] = torch.empty_like(s["lagr"]), torch.empty_like(s["lagr"])
        gen.prepare()
    elif kind in ("lattice", "slab"):
        s["glass"] = 32 if N % 32 == 0 else 16
        s["pos"] = torch.empty((N ** 3, 3), device=DEV)
        s["vel"] = torch.empty((N ** 3, 3), device=DEV)
        gen.prepare()
    elif kind == "potential":
        s["spec"] = _potential_input(N, cfg, seed)
        gen.prepare()
    elif kind == "gradient":
        s["w"] = _noise(N, seed).requires_grad_(True)
        s["alpha"] = torch.tensor(alpha, dtype=torch.float32, device=DEV, requires_grad=True)
        s["g"] = torch.randn((3, N, N, N), generator=_rng(seed, 4), device=DEV)
        gen.prepare()
    return s


def _transform_input(case, seed):
    N, n = case["N"], range(case["fields"])
    return ([torch.randn((N, N, N), generator=_rng(seed, 3 + 10 * i), device=DEV) for i in n],
            [_noise(N, int(seed) + 7919 * i) for i in n])


def _potential_input(N, cfg, seed):
    amp = _factors(cfg, None, "g")["g"]
    return (amp * _noise(N, seed).to(torch.complex128)).to(torch.complex64)


# -------------------------------------------------------------------- pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        return s["gen"].run(s["lagr"], s["pos"], s["vel"])
    if kind in ("lattice", "slab"):
        pos, vel, _ = s["gen"].run_lattice(s["glass"], 100.0, case["N"] // s["glass"], s["pos"], s["vel"])
        return pos, vel
    if kind == "batch":
        s["batch"].run(s["lagr"], s["pos"], s["vel"])
        return s["pos"], s["vel"]
    if kind == "potential":
        s["gen"].set_spectrum(s["spec"])
        s["gen"].stage("modal")
        return s["gen"].spectrum()
    if kind == "gradient":
        d = displacement(s["gen"], s["w"], s["alpha"])
        gw, ga = torch.autograd.grad(d, (s["w"], s["alpha"]), s["g"])
        return d.detach(), gw, ga
    if kind == "transforms":
        return [s["gen"].r2c(x) for x in s["real"]], [s["gen"].c2r(x) for x in s["spec"]]
    return s["basis"].compute_mode_bispectra_covariance(), s["basis"].compute_QS_C(s["S"])


def _fft_flops(N):
    return 2.5 * N ** 3 * math.log2(N ** 3)


def _terms(alpha):
    M = alpha.shape[0]
    t = [(p, q, r) for p in range(M) for q in range(p, M) for r in range(q, M) if alpha[p, q, r] != 0]
    return t, {x for p, q, _ in t for x in (p, q)}, {r for _, _, r in t}


def _modal_flops(N, alpha):
    t, used, rs = _terms(alpha)
    return (len(used) + len(rs)) * _fft_flops(N) + N ** 3 * (3 * len(t) + 4 * len(used) + 10 * len(rs))


def work(case):
    kind = case["kind"]
    if kind == "covariance":
        m, g = case["modes"], case["grid"]
        n, pts = m * (m + 1) * (m + 2) // 6, g ** 3 / 11.6
        return {"bytes": 8.0 * (n * pts + n * n), "flops": n * (n + 1) * pts + 4.0 * n * pts}
    N = case["N"]
    spec, real = 8.0 * N * N * (N // 2 + 1), 4.0 * N ** 3
    if kind == "transforms":
        return {"bytes": case["fields"] * 2 * (spec + real), "flops": case["fields"] * 2 * _fft_flops(N)}
    lpt = 13 * _fft_flops(N) + 60.0 * N ** 3
    if kind == "batch":
        fl = sum(_modal_flops(N, _template(t)[0]) + lpt for t in _batch(case))
        return {"bytes": case["count"] * 36.0 * N ** 3, "flops": fl}
    modal = _modal_flops(N, _template(case["template"])[0])
    if kind == "potential":
        return {"bytes": 2 * spec, "flops": modal}
    if kind == "gradient":
        return {"bytes": 2 * spec + 6 * real, "flops": 3 * (modal + lpt)}
    if kind == "run":
        return {"bytes": 36.0 * case["particles"], "flops": modal + lpt + 100.0 * case["particles"]}
    return {"bytes": 24.0 * N ** 3, "flops": modal + lpt}


# ---------------------------------------------------- the path in 64 bits
def _transfer_table():
    """log10 k, log10 T of the BBKS transfer function the plans are given, T = 1 at its first k."""
    k = np.logspace(-5, 2, 2000)
    q = k / 0.21
    t = np.log(1 + 2.34 * q) / (2.34 * q) * (1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3
                                          + (6.71 * q) ** 4) ** -0.25
    return np.log10(k), np.log10(t) - np.log10(t[0])


def _transfer(k):
    lk, lt = _transfer_table()
    with np.errstate(divide="ignore"):
        x = np.log10(k)
    return np.where((x < lk[0]) | (x > lk[-1]), 0.0, 10.0 ** np.interp(x, lk, lt))


def _romberg(f, a, b):
    """Romberg quadrature as the reference stops it: five estimates, 1e-8 of the value."""
    h, est, trap = [1.0], [], 0.0
    for j in range(40):
        if j == 0:
            trap = 0.5 * (b - a) * float(f(np.array([a]))[0] + f(np.array([b]))[0])
        else:
            n = 1 << (j - 1)
            d = (b - a) / n
            trap = 0.5 * (trap + d * float(np.sum(f(a + d * (np.arange(n) + 0.5)))))
        est.append(trap)
        if j >= 4:  # Neville's tableau at h = 0; its last correction decides
            x, t = h[-5:], est[-5:]
            for m in range(1, 5):
                last = t
                t = [(x[i + m] * last[i] - x[i] * last[i + 1]) / (x[i + m] - x[i]) for i in range(5 - m)]
            if abs(t[0] - last[-1]) <= 1e-8 * abs(t[0]):
                return t[0]
        h.append(0.25 * h[-1])
    return math.nan


def _scalars(cfg):
    """sigma8 normalisation, growth factors, velocity prefactors."""
    Om, OL, ns = cfg["Omega"], cfg["OmegaLambda"], cfg["PrimordialIndex"]

    def sigma2(k):
        kr = np.where(k > 0, 8 * k, 1.0)
        w = 3 * (np.sin(kr) / kr ** 3 - np.cos(kr) / kr ** 2)
        p = np.where(k > 0, k, 1.0) ** ns * _transfer(k) ** 2
        return np.where(8 * k < 1e-8, 0.0, 4 * np.pi * k ** 2 * w ** 2 * p)

    norm = cfg["Sigma8"] ** 2 / _romberg(sigma2, 0.0, 500.0 / 8)

    def growth(a):
        integral = _romberg(lambda x: (x / (Om + (1 - Om - OL) * x + OL * x ** 3)) ** 1.5, 0.0, a)
        return math.sqrt(Om / a ** 3 + (1 - Om - OL) / a ** 2 + OL) * integral

    a = 1 / (1 + cfg["Redshift"])
    D0 = growth(1.0) / growth(1e-8) * 1e-8
    H = 3.2407789e-18 * cfg["UnitLength_in_cm"] / cfg["UnitVelocity_in_cm_per_s"]
    Ha = H * math.sqrt(Om / a ** 3 + (1 - Om - OL) / a ** 2 + OL)
    Oa = Om / (Om + a * (1 - Om - OL) + a ** 3 * OL)
    return dict(norm=norm, D=growth(1.0) / growth(a), beta=1.5 * Om / 2998.0 ** 2 / D0,
                v1=a * Ha * Oa ** 0.6 / math.sqrt(a), v2=a * Ha * 2 * Oa ** (4 / 7) / math.sqrt(a))


def _k(N):
    """Signed wave numbers of the axes; kz = N/2 is taken as positive, as the path's own factors take it."""
    i = torch.arange(N, device=DEV)
    s = torch.where(i < N // 2, i, i - N).to(F64)
    return s[:, None, None], s[None, :, None], torch.arange(N // 2 + 1, device=DEV, dtype=F64)[None, None, :]


def _keep(cfg, k):
    """Cells inside the cut: |k| Box / (2 pi) against Nsample / 2, per axis or on the sphere, in the reference's order
    of roundings, which decide on the boundary itself."""
    h, box = cfg["Nsample"] // 2, cfg["Box"]
    f = [torch.as_tensor(x.cpu().numpy() * 2 * np.pi / box, device=DEV) for x in k]
    if cfg["SphereMode"]:
        return torch.sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]) * box / (2 * np.pi) <= h
    f = [x.abs() * box / (2 * np.pi) <= h for x in f]
    return f[0] & f[1] & f[2]


def _factors(cfg, x0, which):
    """Spectral factors: noise amplitude g on the cells that are drawn, field filters q[n], radial parts r[n]
    (with Fnl / N^3), t = T / (D Beta); the scalars as sc."""
    N, box, ns, sc = cfg["Nmesh"], cfg["Box"], cfg["PrimordialIndex"], _scalars(cfg)
    kF = 2 * np.pi / box
    kx, ky, kz = _k(N)
    n2 = kx ** 2 + ky ** 2 + kz ** 2
    on = _keep(cfg, (kx, ky, kz)) & (n2 > 0)
    kk = kF * torch.sqrt(torch.where(on, n2, 1.0))
    out = {"sc": sc}
    if "g" in which:
        drawn = on & (kx > -N / 2) & (ky > -N / 2) & (kz < N / 2)
        out["g"] = torch.where(drawn, math.sqrt(sc["norm"]) * (2 * np.pi / box) ** 1.5 * sc["beta"] * kk ** (ns / 2 - 2),
                               0.0)
    if "q" in which:
        s = (4 - ns) / 3
        lo, hi = kF ** s, (kF * cfg["Nmax"]) ** s
        kbar = -1 + 2 * (kk ** s - lo) / (hi - lo)
        P = [torch.ones_like(kbar), kbar]
        for l in range(2, len(x0)):
            P.append(((2 * l - 1) * kbar * P[l - 1] - (l - 1) * P[l - 2]) / l)
        out["q"], out["r"] = [], []
        for n in range(len(x0)):
            rad = kk ** (s * (n - 3)) if n <= 3 else (P[n - 1] - float(x0[n - 1])) / kk ** 2
            out["q"].append(torch.where(on, rad * kk ** (4 - ns), 0.0))
            out["r"].append(torch.where(on, cfg["Fnl"] / N ** 3 * rad, 0.0))
    if "t" in which:
        m = np.arange(3 * (N // 2) ** 2 + 1)
        tab = torch.from_numpy(_transfer(kF * np.sqrt(m)) / sc["D"] / sc["beta"]).to(DEV)
        out["t"] = tab[n2.to(torch.int64)]
    return out


def _c2r(x):
    """FFTW's unnormalised c2r: of the kz = 0 and N/2 planes it takes the Hermitian part alone."""
    N = x.shape[0]
    x = x.clone()
    for z in (0, N // 2):
        p = x[:, :, z]
        x[:, :, z] = 0.5 * (p + torch.conj(torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1))))
    return torch.fft.irfftn(x, s=(N, N, N), norm="forward")


def _potential(phi, alpha, F):
    """Total potential of the Gaussian one: phi + sum_r rho_r r2c(sum alpha_pqr f_p f_q), the counter-terms with it."""
    M = alpha.shape[0]
    a = alpha.detach().cpu().numpy() if isinstance(alpha, torch.Tensor) else alpha
    terms, used, _ = _terms(a)
    by = {}
    for p, q, r in terms:
        by.setdefault(r, []).append((p, q, alpha[p, q, r]))
    if M > 2 and a[0, 1, 2] != 0:
        by.setdefault(2, []).append((0, 1, alpha[1, 1, 1]))
        by.setdefault(1, []).append((0, 2, -alpha[1, 1, 1]))
        used |= {0, 1, 2}
    f = {p: _c2r(F["q"][p] * phi) for p in sorted(used)}
    out = phi
    for r in sorted(by):
        out = out + F["r"][r] * torch.fft.rfftn(sum(c * f[p] * f[q] for p, q, c in by[r]))
    return out


def _fields(cfg, phi, twb):
    """psi1 and psi2 / N^3 on the grid."""
    N, box = cfg["Nmesh"], cfg["Box"]
    n3 = float(N) ** 3
    kk = _k(N)
    ka = [2 * np.pi / box * x for x in kk]
    k2 = ka[0] ** 2 + ka[1] ** 2 + ka[2] ** 2
    d = {(a, b): _c2r(-ka[a] * ka[b] * twb * phi) for a in range(3) for b in range(a, 3)}
    S = d[0, 0] * (d[1, 1] + d[2, 2]) + d[1, 1] * d[2, 2] - d[0, 1] ** 2 - d[0, 2] ** 2 - d[1, 2] ** 2
    inv = torch.where(k2 > 0, -1 / torch.where(k2 > 0, k2, 1.0), 0.0)
    Sh = inv * torch.fft.rfftn(S)
    smth = 1.0
    for x in kk:
        smth = smth / torch.sinc(x / N) ** 2
    return ([_c2r(1j * ka[a] * twb * smth * phi) for a in range(3)],
            [_c2r(1j * ka[a] * smth * Sh) / n3 for a in range(3)])


_MASK = (1 << 48) - 1


def _ranlux_words(seeds):
    """Initial words of ranlxd for int64 seeds (zero: one), 12 tensors."""
    v = torch.where(seeds == 0, torch.ones_like(seeds), seeds)
    bits = [(v >> i) & 1 for i in range(31)]
    for n in range(31, 12 * 48):
        bits.append(bits[n - 31] ^ bits[n - 13])
    words = []
    for w in range(12):
        x = torch.zeros_like(v)
        for b in bits[48 * w:48 * w + 48]:
            x = 2 * x + (1 - b)
        words.append(x)
    return words


def _seed_table(seed, N):
    """The N^2 column seeds, drawn from one sequential stream in shells."""
    x = [int(w) for w in _ranlux_words(torch.tensor([seed]))]
    need, c, got = N * N, 0, []
    while len(got) < need:
        for _ in range(16):  # 202 steps = 16 turns of the 12 words and 10 more
            for a, b in ((0, 7), (1, 8), (2, 9), (3, 10), (4, 11), (5, 0), (6, 1), (7, 2), (8, 3), (9, 4), (10, 5),
                         (11, 6)):
                d = x[b] - x[a] - c
                c = 1 if d < 0 else 0
                x[a] = d & _MASK
        for a in range(10):
            d = x[(a + 7) % 12] - x[a] - c
            c = 1 if d < 0 else 0
            x[a] = d & _MASK
        x = x[10:] + x[:10]
        got += x
    u = (np.array(got[:need], dtype=np.float64) / 2.0 ** 48 * float(0x7fffffff)).astype(np.int64)
    t, at = np.zeros((N, N), dtype=np.int64), 0
    for i in range(N // 2):
        e = N - 1 - i
        for line, n in ((t[i, :i], i), (t[:i + 1, i], i + 1), (t[e, :i], i), (t[::-1][:i + 1, i], i + 1),
                        (t[i, ::-1][:i], i), (t[:i + 1, e], i + 1), (t[e, ::-1][:i], i),
                        (t[::-1][:i + 1, e], i + 1)):
            line[:] = u[at:at + n]
            at += n
    return torch.from_numpy(t).to(DEV)


def _gaussian(cfg):
    """Gaussian potential of the parameter file's Seed."""
    N, h = cfg["Nmesh"], cfg["Nmesh"] // 2
    x, c = _ranlux_words(_seed_table(cfg["Seed"], N).reshape(-1)), 0
    u = []
    while len(u) < N:  # two draws for each of the N / 2 cells of a column
        for t in range(202):
            a = t % 12
            d = x[(a + 7) % 12] - x[a] - c
            c = (d < 0).to(torch.int64)
            x[a] = d & _MASK
        x = x[10:] + x[:10]
        u += [w.to(F64) / 2.0 ** 48 for w in x]
    phase = torch.stack(u[0:N:2], 1).reshape(N, N, h) * (2 * math.pi)
    amp = torch.stack(u[1:N:2], 1).reshape(N, N, h)
    full = torch.zeros((N, N, h + 1), dtype=torch.complex128, device=DEV)
    full[:, :, :h] = torch.polar(torch.sqrt(-torch.log(amp)), phase)
    full *= _factors(cfg, None, "g")["g"]
    p = full[:, :, 0].clone()  # kz = 0: half of the plane is drawn, the other half its conjugate
    mirror = torch.conj(torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1)))
    i = torch.arange(N, device=DEV)
    own = (i[:, None] > 0) & (i[:, None] < h) | (i[:, None] == 0) & (i[None, :] < h)
    full[:, :, 0] = torch.where(own, p, mirror)
    full[h, :, 0] = 0
    full[:, h, 0] = 0
    full[0, 0, 0] = 0
    return full


def _read(cfg, sc, psi, lagr):
    """Positions and velocities of particles: trilinear read-out, periodic wrap of the float32 sum."""
    N, box = cfg["Nmesh"], cfg["Box"]
    u = lagr.to(F64) / box * N
    i = u.floor().clamp(0, N - 1)
    f = u - i
    i = i.to(torch.int64)
    out = [torch.zeros_like(u), torch.zeros_like(u)]
    for corner in range(8):
        b = [(corner >> a) & 1 for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (f[:, a] if b[a] else 1 - f[:, a])
        j = [(i[:, a] + b[a]) % N for a in range(3)]
        at = (j[0] * N + j[1]) * N + j[2]
        for o, field in zip(out, psi):
            for a in range(3):
                o[:, a] += w * field[a].reshape(-1)[at]
    d1, d2 = out
    x = lagr.to(F64) + d1 - 3 / 7 * d2
    x = torch.where(x < 0, x + box, x)
    x = torch.where(x.to(torch.float32) >= box, x - box, x).clamp_(min=0.0)
    return x, d1 * sc["v1"] - 3 / 7 * d2 * sc["v2"]


def _realisation(cfg, template, lagr):
    alpha, x0 = _template(template)
    F = _factors(cfg, x0, "qt")
    phi = _potential(_gaussian(cfg), alpha, F)
    return _read(cfg, F["sc"], _fields(cfg, phi, F["t"]), lagr)


def exact(case, seed):
    kind = case["kind"]
    if kind == "covariance":
        kmin, kmax = _grid_case(case, seed)
        return _exact_covariance(case, seed, kmin, kmax)
    N = case["N"]
    if N > 512:
        return None  # its column seeds alone take longer than is wanted
    if kind == "transforms":
        real, spec = _transform_input(case, seed)
        return [torch.fft.rfftn(x.to(F64)) for x in real], [_c2r(x.to(torch.complex128)) for x in spec]
    if kind == "batch":
        got = []
        for i, t in enumerate(_batch(case)):
            cfg = _cfg(case, int(seed) + 7919 * i, t)
            got.append(_realisation(cfg, t, _lattice(N, cfg["Box"])))
        return [p for p, _ in got], [v for _, v in got]
    cfg = _cfg(case, seed)
    alpha, x0 = _template(case["template"])
    if kind == "potential":
        F = _factors(cfg, x0, "q")
        phi = _potential(_potential_input(N, cfg, seed).to(torch.complex128), alpha, F)
        phi[0, 0, 0] = 0
        return phi
    if kind == "gradient":
        F = _factors(cfg, x0, "gqt")
        w = _noise(N, seed).to(torch.complex128).requires_grad_(True)
        a = torch.tensor(alpha, dtype=torch.float32, device=DEV).to(F64).requires_grad_(True)
        psi1, psi2 = _fields(cfg, _potential(F["g"] * w, a, F), F["t"])
        d = torch.stack([x - 3 / 7 * y for x, y in zip(psi1, psi2)])
        g = torch.randn((3, N, N, N), generator=_rng(seed, 4), device=DEV).to(F64)
        gw, _ = torch.autograd.grad(d, (w, a), g)
        return d.detach(), gw, None  # alpha's gradient has entries for absent terms too
    if kind == "run":
        return _realisation(cfg, case["template"], _particles(case, seed, cfg["Box"]))
    g = 32 if N % 32 == 0 else 16
    lagr, t = _lattice(N, cfg["Box"]), N // g
    lagr = lagr.reshape(t, g, t, g, t, g, 3).permute(0, 2, 4, 1, 3, 5, 6).reshape(-1, 3).contiguous()
    return _realisation(cfg, case["template"], lagr)


def _exact_covariance(case, seed, kmin, kmax):
    n, M, s = case["grid"], case["modes"], (4 - BASE["PrimordialIndex"]) / 3
    k = np.linspace(kmin, kmax, n)
    wk = np.where(k > 2 * np.sqrt(kmin * kmax), 1 / np.sqrt(k), 1 / k)
    wk[k < 2 * kmin] = 1 / np.sqrt(k[k < 2 * kmin])
    a, b, c = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    on = (a >= b) & (b >= c)
    a, b, c = a[on], b[on], c[on]
    on = k[b] + k[c] >= k[a]
    a, b, c = a[on], b[on], c[on]
    w = wk[a] * wk[b] * wk[c]
    w = w / w.sum()
    span = kmax ** s - kmin ** s
    at = np.concatenate([-1 + 2 / span * (k ** s - kmin ** s), [-1 - 2 * kmin ** s / span]])
    P = [np.ones(n + 1), at]
    for l in range(2, M):
        P.append(((2 * l - 1) * at * P[-1] - (l - 1) * P[-2]) / l)
    f = np.stack([k ** (2 + s * (p - 3)) if p <= 3 else P[p - 1][:-1] - P[p - 1][-1] for p in range(M)])
    f, w = torch.from_numpy(f).to(DEV), torch.from_numpy(w).to(DEV)
    e = [f[:, torch.from_numpy(x).to(DEV)] for x in (a, b, c)]
    modes = [(p, q, r) for p in range(M) for q in range(p + 1) for r in range(q + 1)]
    Q = torch.empty((len(modes), len(a)), dtype=F64, device=DEV)
    for i, (p, q, r) in enumerate(modes):
        Q[i] = (e[0][p] * (e[1][q] * e[2][r] + e[1][r] * e[2][q]) + e[0][q] * (e[1][p] * e[2][r] + e[1][r] * e[2][p])
                + e[0][r] * (e[1][p] * e[2][q] + e[1][q] * e[2][p])) / 6
    S = torch.from_numpy(_shapes((k[a], k[b], k[c]), seed)).to(DEV)
    return (Q * w) @ Q.T, (S * w) @ Q.T
