"""What a gradient takes from its plan and from its caller: the table of its own
forward pass, whatever table the plan holds by then."""
import numpy as np
import pytest
import torch

from aarambam_gb300.adjoint import displacement, white_noise
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg

pytestmark = pytest.mark.gpu


def generator(N, alpha):
    return ICGenerator(make_cfg(N, 500.0, 3, 100.0, alpha.shape[0], "", 512), alpha, np.linspace(1.0, 0.5, alpha.shape[0]),
                       *bbks())


def symmetric(M, terms):
    a = np.zeros((M, M, M))
    for p, q, r, v in terms:
        for t in ((p, q, r), (p, r, q), (q, p, r), (q, r, p), (r, p, q), (r, q, p)):
            a[t] = v
    return a


def rel(a, b):
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


@pytest.mark.parametrize("N", [16, 256])
def test_backward_after_another_forward(cuda, N):
    """Two forwards on one generator before either backward, the counter-terms
    in one table alone: each gradient is that of a generator of its own."""
    tabs = [symmetric(4, [(0, 0, 3, 1.0), (0, 1, 2, 6.0), (1, 1, 1, -2.0)]), symmetric(4, [(0, 0, 3, -0.5), (1, 1, 1, 3.0)])]
    gd = torch.randn((3, N, N, N), generator=torch.Generator(device="cuda").manual_seed(2), device=cuda)

    def leaves(i):
        return (white_noise(N, 7 + i, cuda).requires_grad_(True),
                torch.tensor(tabs[i], dtype=torch.float64, requires_grad=True))

    want = []
    for i in range(2):
        w, a = leaves(i)
        displacement(generator(N, tabs[i]), w, a).backward(gd)
        want.append((w.grad, a.grad))
    shared = generator(N, tabs[0])
    got = [leaves(i) for i in range(2)]
    disp = [displacement(shared, *got[i]) for i in range(2)]
    disp[0].backward(gd)
    assert np.array_equal(shared.tables[0], tabs[1])  # and the plan still holds the later table
    disp[1].backward(gd)
    for (w, a), (gw, ga) in zip(got, want):
        assert torch.equal(w.grad, gw)
        assert rel(a.grad, ga) < 1e-12  # FP64 sums in another order
