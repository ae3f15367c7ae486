"""The autotuner's candidates: the schedule that the plan runs by itself is
among them, and the report names the blocks that the kernel was compiled for."""
import pytest

from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg, table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,tab,M,minb,threads", [(256, "scalarI_m10_L500_n256", 10, 6, 160),
                                                  (256, "scalarI_m13_L500_n256_mu0p5", 13, 4, 224)])
def test_own_schedule_is_a_candidate(cuda, N, tab, M, minb, threads):
    # rows in pairs: a line per 16 threads, M lines; 64 registers a thread
    g = ICGenerator(make_cfg(N, 500.0, 5, 10.0, M, tab, 256), *table(tab, M), *bbks())
    lines = [l for l in g.autotune().splitlines() if l.strip()]
    assert sum(l.startswith("*") for l in lines) == 1
    own = [l for l in lines if f"rows=nvrtc minb={minb} threads={threads} " in l]
    assert len(own) == 3  # one for each item grouping
    assert len({l[1:].split(" group=")[0] for l in lines}) * 3 == len(lines)  # no shape twice
