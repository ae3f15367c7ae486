"""Conjugate and negated views as inputs: torch keeps both as flags on the
original memory, which the library reads by address."""
import ctypes as C

import numpy as np
import pytest
import torch

import aarambam_gb300.ic as ic
from aarambam_gb300 import _lib
from aarambam_gb300.ic import ICGenerator

N = 4


class Reader:
    """Keeps what stands at the address of the first array argument."""

    def __init__(self, scalars):
        self.n, self.seen = scalars, None

    def __getattr__(self, name):
        def call(h, address, *rest):
            self.seen = np.frombuffer((C.c_float * self.n).from_address(address), np.float32).copy()
            return _lib.AAR_OK
        return call


@pytest.fixture
def generator(monkeypatch):
    monkeypatch.setattr(ic, "_ptr", lambda t: t.data_ptr())
    monkeypatch.setattr(ICGenerator, "_stream", lambda self: None)
    g = ICGenerator.__new__(ICGenerator)
    g.h, g.N, g.device = None, N, torch.device("cpu")
    return g


@pytest.mark.parametrize("name", ["c2r", "set_spectrum"])
def test_a_conjugate_spectrum_is_read_conjugated(generator, name):
    x = torch.randn((N, N, N // 2 + 1), dtype=torch.complex64).conj()
    generator.L = Reader(2 * x.numel())
    getattr(generator, name)(x)
    assert np.array_equal(generator.L.seen.view(np.complex64), x.resolve_conj().numpy().ravel())


@pytest.mark.parametrize("name", ["r2c", "run", "readout"])
def test_a_negated_array_is_read_negated(generator, name):
    x = torch._neg_view(torch.randn((N, N, N) if name == "r2c" else (N, 3)))
    assert x.is_neg()
    generator.L = Reader(x.numel())
    getattr(generator, name)(x)
    assert np.array_equal(generator.L.seen, x.resolve_neg().contiguous().numpy().ravel())
