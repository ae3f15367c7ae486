"""The strided x and y passes with every factor they carry (filters, 2LPT x
and y factors, 1/k^2), at each grid size they are compiled for: the potential
against the plain FP64 form's on the same realisation, the displacement
fields against the 2LPT formulas (main.c:1180-1368) in 64 bits on the plan's
own potential, kz = N/2 taken as positive (the plain form takes it as
negative, as the reference does; the two differ in psi2 on the edges where
two components are at the Nyquist index, 5e-4 of it at N = 16).

Tolerances: a transform pass rounds each value a few times in FP32 (2^-24 =
6e-8); the potential goes through 6 passes and the rows, psi1 through 3, so
1e-6 relative RMS leaves a factor of a few; psi2 is a cancellation of
products of second derivatives and is held to the 2e-4 of the field tests.
"""
import numpy as np
import pytest
import torch

from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg, table

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = a.to(torch.complex128), b.to(torch.complex128)
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


def c2r(x):
    """FFTW's c2r: of the kz = 0 and N/2 planes the Hermitian part counts."""
    N = x.shape[0]
    x = x.clone()
    for z in (0, N // 2):
        p = x[:, :, z]
        x[:, :, z] = 0.5 * (p + torch.conj(torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1))))
    return torch.fft.irfftn(x, s=(N, N, N), norm="forward")


def lpt_fields(g, phi):
    """psi1 and psi2 (before its 1/N^3) of the potential phi, 64 bits."""
    N, box, sc = g.N, g.cfg["Box"], g.scalars
    kF, dev = 2 * np.pi / box, phi.device
    i = torch.arange(N, device=dev)
    s = torch.where(i < N // 2, i, i - N).double()
    k = [s[:, None, None], s[None, :, None], torch.arange(N // 2 + 1, device=dev).double()[None, None, :]]
    n2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    kt, tt = bbks()
    with np.errstate(divide="ignore"):
        lk = np.log10(kF * np.sqrt(np.arange(3 * (N // 2) ** 2 + 1)))
    T = 10.0 ** np.interp(lk, np.log10(kt), np.log10(tt) - np.log10(tt[0]))
    T[0] = 0.0
    twb = torch.from_numpy(T / sc["dplus"] / sc["beta"]).to(dev)[n2.long()]
    sm = 1.0
    for x in k:
        sm = sm / torch.sinc(x / N) ** 2
    d = {(a, b): c2r(-kF * kF * k[a] * k[b] * twb * phi) for a in range(3) for b in range(a, 3)}
    S = d[0, 0] * (d[1, 1] + d[2, 2]) + d[1, 1] * d[2, 2] - d[0, 1] ** 2 - d[0, 2] ** 2 - d[1, 2] ** 2
    Sh = torch.where(n2 > 0, -1 / (kF * kF * torch.clamp(n2, min=1.0)), 0.0) * torch.fft.rfftn(S)
    return [c2r(1j * kF * k[a] * twb * sm * phi) for a in range(3)] + [c2r(1j * kF * k[a] * sm * Sh) for a in range(3)]


@pytest.mark.parametrize("N,sphere,nsample", [(16, 0, 16), (32, 1, 32), (64, 0, 50), (128, 1, 100), (256, 0, 256)])
@pytest.mark.parametrize("tab,M", [("scalarI_m10_L500_n256", 10), ("equil_m9_L500_n256", 9)])
def test_passes_match_plain_fp64(cuda, N, sphere, nsample, tab, M):
    cfg = make_cfg(N, 500.0, 77, 100.0, M, tab, 256, Nsample=nsample, SphereMode=sphere)
    lagr = torch.rand((100, 3), generator=torch.Generator(device="cuda").manual_seed(1), device=cuda) * 499.0
    plain = ICGenerator(cfg, *table(tab, M), *bbks(), precision="fp64_regrouped")
    plain.run(lagr)
    g = ICGenerator(cfg, *table(tab, M), *bbks())
    g.run(lagr)
    assert rel(g.spectrum(), plain.spectrum()) < 1e-6
    for i, want in enumerate(lpt_fields(g, g.spectrum().to(torch.complex128))):
        assert rel(g.field(i), want) < (1e-6 if i < 3 else 2e-4), i


@pytest.mark.parametrize("N", [64, 512])
def test_single_slot_matches_plain_fp64(cuda, N):
    """One active r (an exact Local table): the pass that adds it straight to
    the potential from N = 512 on, the accumulating one below."""
    alpha, x0 = np.zeros((6, 6, 6)), np.linspace(1.0, 0.5, 6)
    for t in ((0, 0, 3), (0, 3, 0), (3, 0, 0)):
        alpha[t] = 1.0
    cfg = make_cfg(N, 500.0, 8, 1000.0, 6, "", 512, Nsample=N - 6)
    lagr = torch.rand((10, 3), generator=torch.Generator(device="cuda").manual_seed(1), device=cuda) * 499.0
    plain = ICGenerator(cfg, alpha, x0, *bbks(), precision="fp64_regrouped")
    plain.run(lagr)
    g = ICGenerator(cfg, alpha, x0, *bbks())
    g.run(lagr)
    assert rel(g.spectrum(), plain.spectrum()) < 1e-6
