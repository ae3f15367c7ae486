"""Device memory of a plan (aar_plan_device_bytes)."""
import numpy as np
import pytest
import torch

from aarambam_gb300.adjoint import displacement, white_noise
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg
from tests.test_gradient_state import symmetric

pytestmark = pytest.mark.gpu


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
