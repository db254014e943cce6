"""What is left after a wait of a flow launch ran out (LBGPU_TEST_GRID_WAIT=1: the grid waits for one block
more than it has, until its limit): the next call that needs the state reports it."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, FP64_FUSED, Box, LbgpuError
from laboetie_gb300 import geometry as geo

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10
NAT = geo.slit(4, 4, 64)
KW = dict(f_ext=(1e-5, 0.0, 0.0))


@pytest.fixture(params=[FP64, FP64_FUSED, FP32_DEV])
def box(request, monkeypatch):
    """A box whose last 20 steps did not reach their end."""
    monkeypatch.setenv("LBGPU_AA_RESIDENT", "grid")
    with Box(NAT, precision=request.param, **KW) as b:
        b.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
        b.flow_steps(20)
        monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
        yield b


def test_equilibration_reports_the_steps_before_it(box):
    _, _, rc = box.equilibration(max_steps=20, check=False)
    assert rc == ERR_TIMEOUT
