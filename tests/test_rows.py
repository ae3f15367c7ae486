"""The modal row kernels (generic and NVRTC; row pairs and, at N = 1024 with
more than 8 lines, folded single rows) against the same row step in 64 bits:
f_p = c2r of each input row, g_r = sum alpha' f_p f_q, r2c of each g_r, for odd
row counts (the last pair has one row), read modes that are not all modes,
and line counts on both sides of the rule between the two kernels.

Tolerance: the row goes through two FP32 transforms of log2 N levels and one
sum of products; 1e-6 of its norm for the transforms (2^-24 sqrt(2 log2 N)
each) and as much for the products.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg

pytestmark = pytest.mark.gpu


def sparse_alpha(M, seed, modes):
    """About 40 sorted triples over `modes`, alpha_012 among them when all of 0, 1, 2 are."""
    r = np.random.default_rng(seed)
    a = np.zeros((M, M, M))
    trip = [tuple(sorted(r.choice(modes, 3))) for _ in range(40)]
    if {0, 1, 2} <= set(modes):
        trip += [(0, 1, 2), (1, 1, 1)]
    for t in trip:
        v = r.uniform(0.5, 1.5)
        for p in {(t[i], t[j], t[k]) for i, j, k in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))}:
            a[p] = v
    return a


def reference(X, alpha):
    """Output rows per active r of the input rows X[p] (complex [M][rows][N/2+1])."""
    M = alpha.shape[0]
    N = 2 * (X.shape[2] - 1)
    X = X.copy()
    X[:, :, [0, -1]] = X[:, :, [0, -1]].real
    f = np.fft.irfft(X, axis=2) * N
    g = {}
    for p in range(M):
        for q in range(p, M):
            for r in range(q, M):
                if alpha[p, q, r]:
                    g[r] = g.get(r, 0) + alpha[p, q, r] * f[p] * f[q]
    if M > 2 and alpha[0, 1, 2]:
        g[2] = g.get(2, 0) + alpha[1, 1, 1] * f[0] * f[1]
        g[1] = g.get(1, 0) - alpha[1, 1, 1] * f[0] * f[2]
    return {r: np.fft.rfft(v, axis=2 - 1) for r, v in g.items()}


@pytest.mark.parametrize("N,M,modes,rows", [
    (16, 5, [0, 1, 2, 3, 4], 7), (32, 9, [0, 1, 2, 5, 8], 33), (64, 10, list(range(10)), 21),
    (128, 32, list(range(32)), 5), (256, 13, list(range(13)), 9), (256, 6, [0, 5], 31), (512, 12, list(range(12)), 3),
    (512, 32, list(range(32)), 4), (1024, 8, list(range(8)), 3), (1024, 9, list(range(9)), 3),
    (1024, 20, list(range(20)), 2), (1024, 32, list(range(32)), 3), (1024, 8, [3], 5)])
@pytest.mark.parametrize("jit", [0, 2])
def test_modal_rows_match_fp64(cuda, N, M, modes, rows, jit):
    alpha = sparse_alpha(M, 17 * N + M, modes)
    g = ICGenerator(make_cfg(N, 500.0, 3, 1.0, M, "", 1024), alpha, np.linspace(1.0, 0.5, M), *bbks())
    assert g.set_jit(jit) == ("on" if jit else "off")
    HP = ((N // 2 + 1) + 7) // 8 * 8
    rng = np.random.default_rng(N + rows)
    X = rng.standard_normal((M, rows, N // 2 + 1)) + 1j * rng.standard_normal((M, rows, N // 2 + 1))
    X = X.astype(np.complex64)
    work = torch.full((M + 1, rows, HP), float("nan"), dtype=torch.complex64, device=cuda)
    work[:M, :, :N // 2 + 1] = torch.from_numpy(X).to(cuda)
    rc = g.L.aar_profile_modal_rows(g.h, C.c_void_p(work.data_ptr()), rows, g._stream())
    assert rc == 0
    torch.cuda.synchronize()
    out = work.cpu().numpy()
    assert np.isnan(out[M]).all()  # nothing beyond the fields
    for r, want in reference(X.astype(np.complex128), alpha).items():
        got = out[r, :, :N // 2 + 1]
        for m in range(rows):  # each row by itself: a pair does not mix its rows
            assert np.linalg.norm(got[m] - want[m]) <= 2e-6 * np.linalg.norm(want[m]), (r, m)
