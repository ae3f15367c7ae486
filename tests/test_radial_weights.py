"""The radial weights rho_r(k) of the modal sum (main.c:825-867) alone: the
ratio of the potential to its 64-bit value over the cells of one |k|^2, where
the transforms' rounding averages out and an error of the weight stays, but for
the gain of the transforms, which is the same at every k (their rounded
twiddles: 2e-7 in any FP32 library) and is taken off.

Tolerance: a weight is at most a product of two table entries rounded from 64
bits (2^-24 each at most, 5e-8 RMS together); a cell's transforms err by 3e-7,
4e-8 over the 60 cells that a |k|^2 has at least: 1e-7 RMS over the |k|^2.
rho_3 = 1 is exact: 5e-8.
"""
import numpy as np
import pytest
import torch

from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg
from tests.test_passes import c2r

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,box,rs", [(128, 500.0, [3]), (128, 500.0, [0]), (128, 500.0, [0, 3, 5]), (256, 500.0, [1, 3]),
                                      (256, 500.0, [0, 5]), (512, 1000.0, [3]), (512, 1000.0, [5]),
                                      (512, 1000.0, [0, 1, 3, 4])])
def test_weights_of_the_modal_sum(cuda, N, box, rs):
    M, ns, nmax = 6, 0.965, max(512, N)
    x0 = np.linspace(1.0, 0.5, M)
    s, kF = (4 - ns) / 3, 2 * np.pi / box
    i = torch.arange(N, device=cuda)
    k1 = torch.where(i < N // 2, i, i - N)
    kz = torch.arange(N // 2 + 1, device=cuda)
    n2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2

    def rho(r, n2):
        k = kF * torch.sqrt(n2.double().clamp(min=1.0))
        if r <= 3:
            return k ** (s * (r - 3))
        kbar = -1 + 2 * (k ** s - kF ** s) / ((kF * nmax) ** s - kF ** s)
        P = [torch.ones_like(kbar), kbar]
        for l in range(2, r):
            P.append(((2 * l - 1) * kbar * P[l - 1] - (l - 1) * P[l - 2]) / l)
        return (P[r - 1] - float(x0[r - 1])) / k ** 2

    alpha = np.zeros((M, M, M))
    c = {}
    for r in rs:  # powers of two that make the slots' parts comparable
        c[r] = 2.0 ** round(-float(torch.log2(rho(r, torch.tensor([(N // 4) ** 2], device=cuda)).abs())))
        alpha[0, 0, r] = alpha[0, r, 0] = alpha[r, 0, 0] = c[r]
    phi = torch.randn((N, N, N // 2 + 1), dtype=torch.complex64,
                      generator=torch.Generator(device="cuda").manual_seed(4), device=cuda)
    g = ICGenerator(make_cfg(N, box, 1, 1.0, M, "", nmax), alpha, x0, *bbks())
    g.set_spectrum(phi)
    g.stage("modal")
    got = g.spectrum().to(torch.complex128)
    phi = phi.to(torch.complex128)
    f = phi.clone()  # q_0 = 1 up to the cut, the whole grid here
    f[0, 0, 0] = 0
    want = torch.fft.rfftn(c2r(f) ** 2) / N ** 3
    want = phi + want * sum(c[r] * rho(r, n2) for r in rs)
    inner = (n2 > 0) & (k1[:, None, None] > -N // 2) & (k1[None, :, None] > -N // 2) & (kz > 0) & (kz < N // 2)
    at = n2[inner]
    num = torch.zeros(int(at.max()) + 1, dtype=torch.float64, device=cuda)
    den, cnt = torch.zeros_like(num), torch.zeros_like(num)
    d = ((got - want) * want.conj()).real[inner]
    num.index_add_(0, at, d)
    den.index_add_(0, at, (want.abs() ** 2)[inner])
    cnt.index_add_(0, at, torch.ones_like(d))
    parts = [c[r] * rho(r, torch.arange(len(num), device=cuda)) for r in rs]
    on = (cnt >= 60) & (sum(parts).abs() > 0.5 * sum(x.abs() for x in parts))  # weights that do not cancel
    assert int(on.sum()) > 500
    err = float((num[on] / den[on]).std())
    print(N, rs, "RMS error of the weight", err)
    assert err < (5e-8 if rs == [3] else 1e-7)
