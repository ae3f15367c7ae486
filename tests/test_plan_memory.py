"""Device memory of a plan (aar_plan_device_bytes, mem_limit_bytes): its fields,
one plane of (N/2+1)^3 filter factors per mode and its tables, and nothing that a
limit counted from them does not cover."""
import numpy as np
import pytest
import torch

from aarambam_gb300.adjoint import displacement, white_noise
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg
from tests.test_gradient_state import symmetric

pytestmark = pytest.mark.gpu

SMALL = 32 * 72 + 16 * 2048  # skip-ahead powers of the generator, the longest term list


def tables_bytes(N, M):
    nsq = 3 * (N // 2) ** 2 + 1
    return 4 * N * N + 12 * N + 8 * N + 4 * nsq * (2 + M + (M + 3) // 4 * 4) + SMALL


@pytest.mark.parametrize("N,M", [(16, 4), (32, 32), (64, 10), (128, 5), (256, 4), (512, 4)])
def test_fused_plan_within_its_fields_filters_and_tables(cuda, N, M):
    alpha = symmetric(M, [(0, 0, 3, 1.0), (0, 1, 2, 6.0), (1, 1, 1, -2.0)])
    ntrip = M * (M + 1) * (M + 2) // 6 + 1
    grad = 16 * 5 + 20 * ntrip  # terms, triples and sums of a gradient
    limit = (8 * N * N * (N // 16 + 1) * 8 * (1 + max(M, 9)) + 4 * M * (N // 2 + 1) ** 3 + tables_bytes(N, M) + grad)
    g = ICGenerator(make_cfg(N, 500.0, 3, 100.0, M, "", 512), alpha, np.linspace(1.0, 0.5, M), *bbks(),
                    mem_limit_bytes=limit)
    g.prepare()
    w = white_noise(N, 7, cuda).requires_grad_(True)
    displacement(g, w, torch.tensor(alpha)).square().sum().backward()
    assert 0 < g.device_bytes <= limit and torch.isfinite(torch.view_as_real(w.grad)).all()


@pytest.mark.parametrize("N", [16, 64, 1024])
def test_plain_plan_holds_its_seed_table_until_it_runs(cuda, N):
    alpha = symmetric(4, [(0, 0, 3, 1.0)])
    limit = 4 * N * N + 32 * 72
    g = ICGenerator(make_cfg(N, 500.0, 3, 100.0, 4, "", 1024), alpha, np.linspace(1.0, 0.5, 4), *bbks(), precision="fp64",
                    mem_limit_bytes=limit)
    assert 0 < g.device_bytes <= limit


@pytest.mark.parametrize("N", [64, 256])
def test_first_gradient_takes_tables_alone(cuda, N):
    """A table that reads one of its modes: the filters that the gradient needs
    besides are there when the plan is prepared."""
    M, alpha = 8, symmetric(8, [(0, 0, 3, 1.0)])
    g = ICGenerator(make_cfg(N, 500.0, 3, 100.0, M, "", 512), alpha, np.linspace(1.0, 0.5, M), *bbks())
    g.prepare()
    held = g.device_bytes
    w = white_noise(N, 7, cuda).requires_grad_(True)
    displacement(g, w, torch.tensor(alpha)).square().sum().backward()
    assert g.device_bytes - held < 4096
    g.set_tables(symmetric(8, [(0, 1, 2, 1.0), (4, 5, 7, 1.0)]))  # other modes read: no other memory
    g.prepare()
    assert g.device_bytes - held < 4096
