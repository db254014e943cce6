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
        b.kind = request.param
        b.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
        b.flow_steps(20)
        monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
        yield b


def test_equilibration_reports_the_steps_before_it(box):
    _, _, rc = box.equilibration(max_steps=20, check=False)
    assert rc == ERR_TIMEOUT


@pytest.mark.parametrize("how", ["init", "set"])
def test_a_new_state_is_not_charged_with_it(box, how):
    if how == "init":
        box.flow_init()
    else:
        w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).reshape(19, 1, 1, 1)
        n = np.ascontiguousarray(w * (NAT == 0))
        box.flow_set(n, n.sum(0), [np.zeros(NAT.shape)] * 3)
    box.sync()
    box.flow_steps(20)
    box.sync()
    assert np.isfinite(box.flow_get()[0]).all()


def gone(box):
    """No call hands out or goes on from the state."""
    for call in (box.flow_get, lambda: box.flow_steps(4), lambda: box.equilibration(max_steps=4), lambda: box.mp_init(Db=0.01)):
        with pytest.raises(LbgpuError):
            call()


def test_the_state_is_gone_once_reported(box):
    with pytest.raises(LbgpuError) as e:
        box.flow_get()
    assert e.value.status == ERR_TIMEOUT
    gone(box)
    box.flow_init()
    box.flow_steps(20)
    box.flow_get()


def test_the_state_is_gone_after_a_loop(box, monkeypatch):
    box.flow_init()
    monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
    _, _, rc = box.equilibration(max_steps=20, check=False)
    monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
    assert rc == ERR_TIMEOUT
    gone(box)


def test_calls_without_the_flow_state_do_not_report_it(box):
    if box.kind != FP32_DEV:
        w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).reshape(19, 1, 1, 1)
        n = np.ascontiguousarray(w * (NAT == 0))
        z = [np.zeros(NAT.shape)] * 3
        box.bounce_back_stream(box.collide(n, n.sum(0), z, z))
    box.pnp_init(bjl=0.4, sigma=0.0)
    box.pnp_set(*box.pnp_get())
    with pytest.raises(LbgpuError) as e:
        box.flow_get()
    assert e.value.status == ERR_TIMEOUT
