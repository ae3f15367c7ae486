"""What a gradient takes from its plan and from its caller: the table of its own
forward pass, whatever table the plan holds by then, scratch that its 16-byte
copies can read, and nothing that another gradient of the plan writes."""
import threading

import numpy as np
import pytest
import torch

from aarambam_gb300 import _lib
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


def gradient(g, phig, phi, gd, scratch, gw, galpha):
    return g.L.aar_adj_gradient(g.h, *(t.data_ptr() for t in (phig, phi, gd, gw, galpha, scratch)), scratch.numel(),
                                g._stream())


def test_misaligned_scratch_is_refused(cuda):
    """On the host, before anything is launched."""
    N = 16
    g = generator(N, symmetric(4, [(0, 0, 3, 1.0)]))
    phi, gd = white_noise(N, 7, cuda), torch.randn((3, N, N, N), device=cuda)
    gw, galpha = torch.zeros_like(phi), torch.zeros((4, 4, 4), dtype=torch.float64, device=cuda)
    need = g.L.aar_adj_gradient_scratch_bytes(g.h)
    scratch = torch.empty(need + 16, dtype=torch.uint8, device=cuda)
    assert gradient(g, phi, phi, gd, scratch[8:], gw, galpha) == _lib.AAR_ERR_ARG
    assert b"16-byte" in g.L.aar_last_error(g.h)
    torch.cuda.synchronize()
    assert not gw.any() and not galpha.any()
    assert gradient(g, phi, phi, gd, scratch[16:], gw, galpha) == _lib.AAR_OK
    torch.cuda.synchronize()
    assert gw.any() and galpha.any()


def test_gradients_of_one_plan_on_two_streams(cuda):
    """Buffers and scratch of their own: what they give one after the other, the
    sums of alpha's gradient (atomic adds in FP64) to the order of summation."""
    N, alpha = 64, symmetric(4, [(0, 0, 3, 1.0), (0, 1, 2, 6.0), (1, 1, 1, -2.0)])
    g = generator(N, alpha)
    need = g.L.aar_adj_gradient_scratch_bytes(g.h)

    def buffers(i):
        phi, gen = white_noise(N, 7 + i, cuda), torch.Generator(device="cuda").manual_seed(2 + i)
        return [phi, phi, torch.randn((3, N, N, N), generator=gen, device=cuda),
                torch.empty(need, dtype=torch.uint8, device=cuda), torch.zeros_like(phi),
                torch.zeros((4, 4, 4), dtype=torch.float64, device=cuda)]

    want = [buffers(i) for i in range(2)]
    for b in want:
        assert gradient(g, *b) == _lib.AAR_OK
    torch.cuda.synchronize()
    got, streams = [buffers(i) for i in range(2)], [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(5):
        for b, s in zip(got, streams):
            with torch.cuda.stream(s):
                assert gradient(g, *b) == _lib.AAR_OK
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a[4], b[4]) and rel(a[5], b[5]) < 1e-12


def test_gradients_of_two_plans_in_two_threads(cuda):
    """Plans of one grid size whose products take different amounts of shared
    memory, each thread on a stream of its own: every launch goes through."""
    N, full = 16, np.zeros((20, 20, 20))
    for p in range(20):
        for q in range(p, 20):
            full[p, q, q:] = 1.0
    rc = [[], []]

    def work(i, g, bufs, stream):
        with torch.cuda.stream(stream):
            for _ in range(400):
                rc[i].append(gradient(g, *bufs))

    threads = []
    for i, alpha in enumerate((symmetric(4, [(0, 0, 3, 1.0)]), full)):
        g, phi, M = generator(N, alpha), white_noise(N, 7, cuda), alpha.shape[0]
        bufs = [phi, phi, torch.randn((3, N, N, N), device=cuda),
                torch.empty(g.L.aar_adj_gradient_scratch_bytes(g.h), dtype=torch.uint8, device=cuda),
                torch.zeros_like(phi), torch.zeros((M, M, M), dtype=torch.float64, device=cuda)]
        assert gradient(g, *bufs) == _lib.AAR_OK
        threads.append(threading.Thread(target=work, args=(i, g, bufs, torch.cuda.Stream())))
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert len(rc[0]) == len(rc[1]) == 400 and not any(rc[0]) and not any(rc[1])
