"""FP64 boxes stepped by one launch for many steps (a node per thread, or four warps per node) against one
launch per step: bit for bit, strict and fused, at the edges of both forms, for fixed steps and for the
reference loop with its force switch, exit and caps.  (The launch-per-step kernel and, in the other test
files, these ones are compared with the oracle.)"""
import numpy as np
import pytest

from laboetie_gb300 import FP64, FP64_FUSED, Box, LbgpuError
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import ERR_NEGATIVE_POPULATION, ERR_STEP_CAP

from test_flow_resident_gpu import box_with, same

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10


def run(monkeypatch, mode, nat, precision, what, **kw):
    monkeypatch.setenv("LBGPU_F64_RESIDENT", mode)
    with Box(nat, precision=precision, **kw) as box:
        out = what(box)
        n, rho, j = box.flow_get()
    return out, n, rho, j


FORMS = [(FP64, "1"), (FP64, "whole"), (FP64_FUSED, "1")]
FORCES = [(1e-5, 0.0, 0.0), (0.0, 2e-5, 0.0), (0.0, 0.0, 1e-5), (1e-5, -2e-5, 3e-6), (0.0, 0.0, 0.0)]


# four warps per node to 152 * 32 = 4864 nodes, a node per thread to 152 * 256 = 38912
@pytest.mark.parametrize("precision,mode", FORMS)
@pytest.mark.parametrize("nf", [1, 31, 32, 33, 4864, 4865, 20000, 38912, 38913])
def test_fixed_steps_and_loop(monkeypatch, precision, mode, nf):
    nat = box_with(nf, nf + 3)
    kw = dict(relaxation_time=1.0 if nf % 2 else 0.83, f_ext=FORCES[nf % 5])

    def what(box):
        box.flow_init()
        box.flow_steps(5)
        box.flow_steps(4, force_on=False)
        box.flow_get(populations=False)
        box.flow_steps(9)
        return box.equilibration(max_steps=9, hist_cap=9, check=False)
    same(run(monkeypatch, "0", nat, precision, what, **kw), run(monkeypatch, mode, nat, precision, what, **kw))


@pytest.mark.parametrize("precision,mode", FORMS)
@pytest.mark.parametrize("f_ext", FORCES)
@pytest.mark.parametrize("tau", [1.0, 0.7])
def test_loop_from_rest(monkeypatch, precision, mode, f_ext, tau):
    nat = box_with(900, 5)
    kw = dict(relaxation_time=tau, f_ext=f_ext)

    def what(box):
        box.flow_init()
        r = box.equilibration(max_steps=25, hist_cap=25, check=False)
        box.flow_steps(6)
        return r
    a, b = run(monkeypatch, "0", nat, precision, what, **kw), run(monkeypatch, mode, nat, precision, what, **kw)
    same(a, b)
    assert b[0][2] == (ERR_STEP_CAP if any(f_ext) else 0)


@pytest.mark.parametrize("precision,mode", FORMS)
@pytest.mark.parametrize("cap", [0, 4, 3])
def test_switch_and_exit(monkeypatch, precision, mode, cap):
    nat = geo.slit(3, 4, 20)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    n = w[:, None, None, None] * (1 + 1e-3 * np.random.default_rng(2).standard_normal((19,) + nat.shape)) * (nat == 0)
    rho, j = n.sum(0), [np.zeros(nat.shape)] * 3

    def what(box):
        box.flow_set(n, rho, j)
        r = box.equilibration(max_steps=cap or 20000, hist_cap=20000, check=False)
        box.flow_steps(8)
        return r
    kw = dict(relaxation_time=0.9, f_ext=(1e-4, 0.0, 0.0), target_error=3e-5)
    a, b = run(monkeypatch, "0", nat, precision, what, **kw), run(monkeypatch, mode, nat, precision, what, **kw)
    same(a, b)
    if not cap:
        assert b[0][2] == 0 and b[0][0] > 10


@pytest.mark.parametrize("precision,mode", FORMS)
def test_negative_population(monkeypatch, precision, mode):
    nat = geo.slit(4, 4, 12)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    n = (w[:, None, None, None] * (nat == 0)).copy()
    n[5, 6, 2, 2] = -0.2
    rho, j = n.sum(0), [np.zeros(nat.shape)] * 3

    def what(box):
        box.flow_set(n, rho, j)
        return box.equilibration(max_steps=50, hist_cap=50, check=False)
    kw = dict(relaxation_time=1.7, f_ext=(1e-5, 0.0, 0.0))
    a, b = run(monkeypatch, "0", nat, precision, what, **kw), run(monkeypatch, mode, nat, precision, what, **kw)
    same(a, b)
    assert b[0][2] == ERR_NEGATIVE_POPULATION


def test_wait_runs_out(monkeypatch):
    nat = geo.slit(4, 4, 64)
    with Box(nat, f_ext=(1e-5, 0.0, 0.0)) as box:
        box.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
        assert box.equilibration(max_steps=20, check=False)[2] == ERR_TIMEOUT
        box.flow_init()
        box.flow_steps(20)
        with pytest.raises(LbgpuError) as e:
            box.flow_get()
        assert e.value.status == ERR_TIMEOUT
        monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
        box.flow_init()
        box.flow_steps(20)
        assert np.isfinite(box.flow_get()[1]).all()
