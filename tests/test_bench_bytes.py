"""bench.py's byte counts of the modal kernels follow the modes that the
products read, as the kernels do."""
import numpy as np
import pytest

import bench


@pytest.mark.parametrize("workload,Q", [("local_m8_n128", 3), ("scalarI_m12_n512", 12), ("scalarI_m20_n1024", 20)])
def test_bytes_follow_the_modes_read(workload, Q):
    cfg = bench.make_cfg(workload, 1)
    alpha = bench.load_tables(cfg["table"], cfg["N_modes"])[0]
    N, R = cfg["Nmesh"], bench.active_r(alpha)
    F = 8.0 * N * N * (N // 2 + 1)
    assert bench.read_modes(alpha) == Q
    for name, fields in (("modal_xinv", 1 + Q), ("modal_ypass_inv", 2 * Q), ("modal_rows", Q + R)):
        assert bench.alg_bytes(name, N, bench.read_modes(alpha), R, 0) == fields * F
    assert bench.path_bytes(N, bench.read_modes(alpha)) == 4.0 * N ** 3 * (46 + 9 * Q)


def test_counter_terms_read_the_first_three():
    alpha = np.zeros((6, 6, 6))
    alpha[4, 4, 5] = 1.0
    assert bench.read_modes(alpha) == 1
    alpha[0, 1, 2] = 1.0
    assert bench.read_modes(alpha) == 4
    alpha[5, 4, 3] = 1.0  # not sorted: not read
    assert bench.read_modes(alpha) == 4
