"""The differentiable chain in one call each way (aar_adj_displacement,
aar_adj_gradient) against the same chain composed from the C ABI's building
blocks (aar_adj_spectral, aar_adj_source, aar_adj_products, the plan's stages
and transforms), whose gradients test_adjoint.py holds to FP64: tables with
modes that no product reads, one mode, 32 modes, cuts, and every grid size.

Tolerance: both sides round each of about 30 FP32 passes once or twice (6e-8
each) in another order, and psi2's source cancels a digit: 2e-5 relative norm.
"""
import numpy as np
import pytest
import torch

from aarambam_gb300.adjoint import (CT, CT_INV_W, CT_W, FWD, GAUSS, HESS, ONE, PSI1, PSI2, Q, RHO, _Ops, displacement,
                                    white_noise)
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg, table
from tests.test_rows import sparse_alpha

pytestmark = pytest.mark.gpu


def composed(gen, w, gdisp):
    ops, N, M = _Ops(gen), gen.N, gen.n_modes
    c2 = -(3.0 / 7.0) / float(N) ** 3
    phig = ops.spec(GAUSS, 0, FWD, w)
    ops.set_spectrum(phig)
    gen.stage("modal")
    phi = gen.spectrum()
    gen.stage("lpt")
    f = [gen.field(i) for i in range(6)]
    disp = torch.stack(f[:3]) + c2 * torch.stack(f[3:])
    gphi, gsrc = torch.zeros_like(phi), torch.zeros_like(phi)
    for a in range(3):
        ops.spec(PSI1, a, CT_W, ops.r2c(gdisp[a]), out=gphi)
        ops.spec(PSI2, a, CT_W, ops.r2c(c2 * gdisp[a]), out=gsrc)
    gS = ops.c2r(ops.spec(ONE, 0, CT_INV_W, gsrc))
    gd = ops.source_adj(torch.stack([ops.c2r(ops.spec(HESS, ab, FWD, phi)) for ab in range(6)]), gS)
    for ab in range(6):
        ops.spec(HESS, ab, CT_W, ops.r2c(gd[ab]), out=gphi)
    gg = torch.stack([ops.c2r(ops.spec(RHO, r, CT_INV_W, gphi)) for r in range(M)])
    ff = torch.stack([ops.c2r(ops.spec(Q, p, FWD, phig)) for p in range(M)])
    gf, ga = ops.products_adj(ff, gg)
    for p in range(M):
        ops.spec(Q, p, CT_W, ops.r2c(gf[p]), out=gphi)
    return disp, ops.spec(GAUSS, 0, CT, gphi), ga


def rel(a, b):
    a, b = a.to(torch.complex128), b.to(torch.complex128)
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


def one_term(M):
    a = np.zeros((M, M, M))
    for t in ((0, 0, M - 1), (0, M - 1, 0), (M - 1, 0, 0)):
        a[t] = 1.0
    return a


@pytest.mark.parametrize("N,M,alpha,sphere,nsample", [
    (16, 4, one_term(4), 0, 16), (32, 32, sparse_alpha(32, 5, list(range(32))), 1, 30), (64, 9, "equil_m9_L500_n256", 0, 64),
    (128, 10, "scalarI_m10_L500_n256", 0, 100), (256, 6, one_term(6), 1, 256), (32, 1, np.ones((1, 1, 1)), 0, 32),
    (512, 4, one_term(4), 0, 512)])
def test_chain_matches_building_blocks(cuda, N, M, alpha, sphere, nsample):
    x0 = np.linspace(1.0, 0.5, M)
    if isinstance(alpha, str):
        alpha, x0 = table(alpha, M)
    cfg = make_cfg(N, 500.0, 3, 100.0, M, "", 512, Nsample=nsample, SphereMode=sphere)
    gen = ICGenerator(cfg, alpha, x0, *bbks())
    w = white_noise(N, 7, cuda)
    gdisp = torch.randn((3, N, N, N), generator=torch.Generator(device="cuda").manual_seed(2), device=cuda)
    wt = w.clone().requires_grad_(True)
    at = torch.tensor(alpha, dtype=torch.float64, requires_grad=True)
    disp = displacement(gen, wt, at)
    fields = [gen.field(i) for i in (0, 5)]
    spec = gen.spectrum()
    disp.backward(gdisp)
    # the plan's fields and spectrum are what the forward pass left
    assert all(torch.equal(gen.field(i), f) for i, f in zip((0, 5), fields)) and torch.equal(gen.spectrum(), spec)
    rdisp, rgw, rga = composed(gen, w, gdisp)
    assert rel(disp.detach(), rdisp) < 2e-6
    assert rel(wt.grad, rgw) < 2e-5
    assert rel(at.grad, rga.cpu()) < 2e-5
    assert torch.equal(at.grad != 0, rga.cpu() != 0)
    assert torch.count_nonzero(wt.grad[rgw == 0]) == 0


@pytest.mark.parametrize("N,M,alpha", [(16, 4, one_term(4)), (64, 5, sparse_alpha(5, 3, [0, 2, 4])), (256, 4, one_term(4))])
def test_memory_limit_changes_no_bit(cuda, N, M, alpha):
    """A plan with a memory limit keeps no transfer cube and all modes' planes
    in the filter cube: the same factors from other places."""
    def results(limit):
        gen = ICGenerator(make_cfg(N, 500.0, 3, 100.0, M, "", 512), alpha, np.linspace(1.0, 0.5, M), *bbks(),
                          mem_limit_bytes=limit)
        w = white_noise(N, 7, cuda).requires_grad_(True)
        disp = displacement(gen, w, torch.tensor(alpha, dtype=torch.float64))
        disp.square().sum().backward()
        return disp.detach(), gen.spectrum(), w.grad
    assert all(torch.equal(a, b) for a, b in zip(results(0), results(1 << 40)))
