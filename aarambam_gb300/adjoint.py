"""Differentiable fused path: white noise -> Gaussian potential -> modal
non-Gaussian potential -> ZA + 2LPT displacement field, as a
torch.autograd.Function with a hand-written adjoint.

`displacement(gen, w_hat, alpha)` returns the displacement field on the grid,
float32 [3, N, N, N]:

    disp_a = psi1_a - (3/7) psi2_a / N^3

with psi1 / psi2 the ZA and 2LPT fields exactly as the path reads them out
at the particles (Aarambam/LPT/Basis/main.c:1486-1507: Pos += dis - 3/7 dis2,
dis2 /= N^3).  Inputs:
  w_hat  complex64 [N, N, N/2+1]: the unit-variance noise whose scaled copy
         amp(k) w_hat is the Gaussian potential (the reference draws
         w = sqrt(-ln u2) e^{2 pi i u1}, main.c:396-459);
  alpha  float64 [M, M, M]: the coefficient table; entries with p <= q <= r
         are the ones the path reads (the reference symmetrises the
         AlphaTable rows, main.c:233-241), and the gradient is returned there.

The backward pass is the transpose of every step (aarambam_gb300/csrc/
chain.cuh); it runs the plan's own FFT passes and recomputes the M filtered
fields f_p and the six Hessians from the saved spectra instead of storing them
(memory: the Gaussian and the total potential spectra are saved; the backward
holds max(2M, 9) + 2 fields of scratch).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib
from ._lib import check
from .ic import ICGenerator, _dense, _ptr

ONE, GAUSS, Q, RHO = _lib.AAR_ADJ_OP_ONE, _lib.AAR_ADJ_OP_GAUSS, _lib.AAR_ADJ_OP_Q, _lib.AAR_ADJ_OP_RHO
HESS, PSI1, PSI2 = _lib.AAR_ADJ_OP_HESS, _lib.AAR_ADJ_OP_PSI1, _lib.AAR_ADJ_OP_PSI2
FWD, CT_W, CT_INV_W, CT = 0, 1, 2, 3  # factor modes: F, conj(F) w, conj(F)/w, conj(F)


class _Ops:
    """Thin wrappers over the plan's C-ABI building blocks."""

    def __init__(self, gen: ICGenerator):
        self.g = gen
        self.L = gen.L
        self.N = gen.N

    def stream(self):
        return C.c_void_p(torch.cuda.current_stream(self.g.device).cuda_stream)

    def spec(self, op, comp, mode, x, out=None):
        acc = out is not None
        if out is None:
            out = torch.empty_like(x)
        check(self.L, self.g.h, self.L.aar_adj_spectral(self.g.h, op, comp, mode, _ptr(x), _ptr(out), int(acc),
                                                        self.stream()))
        return out

    def c2r(self, x):
        return self.g.c2r(x)

    def r2c(self, x):
        return self.g.r2c(x)

    def set_spectrum(self, x):
        check(self.L, self.g.h, self.L.aar_set_spectrum(self.g.h, _ptr(x), self.stream()))

    def source_adj(self, d, gS):
        out = torch.empty_like(d)
        check(self.L, self.g.h, self.L.aar_adj_source(self.g.h, _ptr(d), _ptr(gS), _ptr(out), self.stream()))
        return out

    def products_adj(self, f, gg):
        M = f.shape[0]
        gf = torch.empty_like(f)
        ga = torch.zeros((M, M, M), dtype=torch.float64, device=f.device)
        check(self.L, self.g.h, self.L.aar_adj_products(self.g.h, _ptr(f), _ptr(gg), _ptr(gf), _ptr(ga),
                                                        self.stream()))
        return gf, ga


class _Displacement(torch.autograd.Function):
    @staticmethod
    def forward(ctx, w_hat, alpha, gen):
        N = gen.N
        ctx.w_dtype = w_hat.dtype
        w_hat = _dense(w_hat, torch.complex64)
        gen.set_tables(alpha.detach().double().cpu().numpy())
        phig, phi = torch.empty_like(w_hat), torch.empty_like(w_hat)
        disp = torch.empty((3, N, N, N), dtype=torch.float32, device=gen.device)
        check(gen.L, gen.h, gen.L.aar_adj_displacement(gen.h, _ptr(w_hat), _ptr(disp), _ptr(phig), _ptr(phi),
                                                       gen._stream()))
        ctx.gen, ctx.tables = gen, gen.tables
        ctx.save_for_backward(phig, phi)
        ctx.alpha_dtype, ctx.alpha_device = alpha.dtype, alpha.device
        return disp

    @staticmethod
    def backward(ctx, gdisp):
        gen = ctx.gen
        phig, phi = ctx.saved_tensors
        gdisp = _dense(gdisp, torch.float32)
        gw = torch.empty_like(phig)
        # at the forward pass's tables, which a later forward pass may have
        # replaced in the plan; the plan goes back to those it holds now
        held = gen.tables
        gen.set_tables(*ctx.tables)
        try:
            M = gen.n_modes
            galpha = torch.empty((M, M, M), dtype=torch.float64, device=gdisp.device)
            scratch = torch.empty(gen.L.aar_adj_gradient_scratch_bytes(gen.h), dtype=torch.uint8, device=gdisp.device)
            check(gen.L, gen.h, gen.L.aar_adj_gradient(gen.h, _ptr(phig), _ptr(phi), _ptr(gdisp), _ptr(gw),
                                                       _ptr(galpha), _ptr(scratch), scratch.numel(), gen._stream()))
        finally:
            gen.set_tables(*held)
        return gw.to(ctx.w_dtype), galpha.to(device=ctx.alpha_device, dtype=ctx.alpha_dtype), None


def displacement(gen: ICGenerator, w_hat: torch.Tensor, alpha: torch.Tensor) -> torch.Tensor:
    """Differentiable displacement field float32 [3, N, N, N] (see the module
    docstring); gradients flow to w_hat and alpha."""
    return _Displacement.apply(w_hat, alpha, gen)


def white_noise(N: int, seed: int, device) -> torch.Tensor:
    """Unit-variance complex noise of the shape the path takes (torch's
    generator; for tests and examples)."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    u1 = torch.rand((N, N, N // 2 + 1), generator=g, dtype=torch.float64)
    u2 = 1.0 - torch.rand((N, N, N // 2 + 1), generator=g, dtype=torch.float64)
    w = torch.sqrt(-torch.log(u2)) * torch.exp(2j * np.pi * u1)
    return w.to(torch.complex64).to(device)
