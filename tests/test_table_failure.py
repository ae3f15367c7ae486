"""What a plan holds after other tables: after a set_tables that ran out of
memory half way it refuses to compute until tables are set again, and then gives
what it gave before; fields that more modes have moved are not handed out."""
import numpy as np
import pytest
import torch

from aarambam_gb300._lib import AarError
from aarambam_gb300.ic import ICGenerator
from tests.common import bbks, make_cfg
from tests.test_gradient_state import symmetric

pytestmark = pytest.mark.gpu


def plan(N, M, limit=0):
    return ICGenerator(make_cfg(N, 500.0, 3, 100.0, M, "", 512), symmetric(M, [(0, 0, 3, 1.0)]), np.linspace(1.0, 0.5, M),
                       *bbks(), mem_limit_bytes=limit)


@pytest.mark.parametrize("spare", [0.0, 0.5])
def test_plan_after_tables_that_did_not_fit(cuda, spare):
    """No room for the filter table of 32 modes, and room for it but not for the
    radial one beside it."""
    N = 32
    nsq = 3 * (N // 2) ** 2 + 1
    whole = plan(N, 4, 1 << 40)
    whole.prepare()
    free = whole.device_bytes - 2 * 4 * 4 * nsq  # what stays when the tables of four modes go
    g = plan(N, 4, free + int((1 + spare) * 4 * 32 * nsq) - 4)
    lagr = torch.rand((1000, 3), generator=torch.Generator(device="cuda").manual_seed(1), device=cuda) * 499.0
    pos, vel = g.run(lagr)
    held = g.device_bytes
    with pytest.raises(AarError):
        g.set_tables(symmetric(32, [(0, 0, 31, 1.0)]), np.linspace(1.0, 0.5, 32))
    with pytest.raises(AarError, match="tables not set"):
        g.run(lagr)
    g.set_tables(symmetric(4, [(0, 0, 3, 1.0)]), np.linspace(1.0, 0.5, 4))
    again = g.run(lagr)
    assert torch.equal(again[0], pos) and torch.equal(again[1], vel)
    assert g.device_bytes == held


def test_fields_are_gone_with_their_memory(cuda):
    g = plan(32, 4)
    for stage in ("noise", "modal", "lpt"):
        g.stage(stage)
    g.field(0)
    g.set_tables(symmetric(16, [(0, 0, 3, 1.0)]), np.linspace(1.0, 0.5, 16))  # more work fields than before
    g.prepare()
    with pytest.raises(AarError, match="run the field stages first"):
        g.field(0)
    g.stage("lpt")
    g.field(0)
