"""Grid sizes at which a kernel takes another path: columns that leave the last
noise warp short, the 1024-point passes with one slot and with several, the
gradient at 1024^3."""
import numpy as np
import pytest
import torch

from aarambam_gb300._lib import check
from aarambam_gb300.adjoint import displacement
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg
from tests.test_chain import composed, one_term, rel
from tests.test_radial_weights import test_weights_of_the_modal_sum as weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,S,sphere", [(8, 2, 0), (12, 3, 1), (20, 5, 0), (132, 6, 0), (132, 6, 1), (164, 4, 0)])
def test_noise_of_grids_off_the_warp(cuda, N, S, sphere):
    """N^2 columns not a multiple of a warp's 8, 16 or 32: the Gaussian spectrum in
    the plan's row order and in the caller's, per cell within the 2e-6 of the FP32
    amplitudes, zero in the same cells."""
    cfg = make_cfg(N, 500.0, 77, 0.0, 4, "", 256, SphereMode=sphere)
    alpha, x0 = one_term(4), np.linspace(1.0, 0.5, 4)

    def gauss(g, dtype):
        out = torch.full((N, N, N // 2 + 1), 7.0, dtype=dtype, device=cuda)
        check(g.L, g.h, g.L.aar_gaussian_spectrum_noalloc(g.h, out.data_ptr(), g._stream()))
        return out

    want = gauss(ICGenerator(cfg, alpha, x0, *bbks(), precision="fp64"), torch.complex128)
    g = ICGenerator(cfg, alpha, x0, *bbks(), precision="slab_fp32", nslab=S)
    g.run(torch.zeros((1, 3), device=cuda))
    for got in (gauss(g, torch.complex64), g.spectrum()):
        assert torch.equal(got == 0, want == 0)
        on = want != 0
        assert float(((got[on] - want[on]).abs() / want[on].abs()).max()) < 2e-6


@pytest.mark.parametrize("rs", [[3], [0], [0, 1, 3]])
def test_weights_1024(cuda, rs):
    weights(cuda, 1024, 1000.0, rs)
    torch.cuda.empty_cache()


def test_chain_1024(cuda):
    N, M = 1024, 4
    alpha = one_term(M)
    gen = ICGenerator(make_cfg(N, 500.0, 3, 100.0, M, "", 1024), alpha, np.linspace(1.0, 0.5, M), *bbks())
    w = torch.randn((N, N, N // 2 + 1), dtype=torch.complex64, generator=torch.Generator(device="cuda").manual_seed(7),
                    device=cuda)
    gdisp = torch.randn((3, N, N, N), generator=torch.Generator(device="cuda").manual_seed(2), device=cuda)
    wt = w.clone().requires_grad_(True)
    at = torch.tensor(alpha, dtype=torch.float64, requires_grad=True)
    disp = displacement(gen, wt, at)
    disp.backward(gdisp)
    torch.cuda.empty_cache()
    rdisp, rgw, rga = composed(gen, w, gdisp)

    def close(a, b):  # rel, a plane at a time
        d = n = 0.0
        for x, y in zip(a, b):
            d += float(torch.linalg.vector_norm(x.to(torch.complex128) - y.to(torch.complex128)) ** 2)
            n += float(torch.linalg.vector_norm(y.to(torch.complex128)) ** 2)
        return (d / n) ** 0.5

    assert close(disp.detach().reshape(-1, N, N), rdisp.reshape(-1, N, N)) < 2e-6
    assert close(wt.grad, rgw) < 2e-5
    assert rel(at.grad, rga.cpu()) < 2e-5
    del rdisp, rgw, disp, wt, gdisp, w
    torch.cuda.empty_cache()
