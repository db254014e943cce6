"""One block of a many-step launch gives up at a rendezvous that all the others pass
(LBGPU_TEST_GRID_WAIT=k: the last block, at the rendezvous k - 1), the launch's last one or an earlier one:
the call reports it, although the first block, which writes the control block, has seen nothing."""
import math

import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, FP64_FUSED, Box, LbgpuError
from laboetie_gb300 import geometry as geo

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10
NAT = geo.slit(4, 4, 64)
KW = dict(f_ext=(1e-5, 0.0, 0.0))
# rendezvous of a loop of two steps: FP64 one a step; FP32 one more before the first
LAST = {FP64: 2, FP64_FUSED: 2, FP32_DEV: 3}


@pytest.mark.parametrize("precision", [FP64, FP64_FUSED, FP32_DEV])
@pytest.mark.parametrize("back", [0, 1])
def test_loop(monkeypatch, precision, back):
    monkeypatch.setenv("LBGPU_AA_RESIDENT", "grid")
    with Box(NAT, precision=precision, **KW) as box:
        box.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", str(LAST[precision] - back + 1))
        _, _, rc = box.equilibration(max_steps=2, check=False)
        assert rc == ERR_TIMEOUT
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", str(LAST[precision] + 2))   # beyond the last: nothing
        box.flow_init()
        steps, _, rc = box.equilibration(max_steps=2, check=False)
        assert rc != ERR_TIMEOUT and steps == 2


@pytest.mark.parametrize("precision", [FP64, FP64_FUSED, FP32_DEV])
def test_fixed_steps(monkeypatch, precision):
    monkeypatch.setenv("LBGPU_AA_RESIDENT", "grid")
    with Box(NAT, precision=precision, **KW) as box:
        box.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "20")   # 20 steps have 19 rendezvous
        box.flow_steps(20)
        with pytest.raises(LbgpuError) as e:
            box.sync()
        assert e.value.status == ERR_TIMEOUT


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_tracer(monkeypatch, precision):
    monkeypatch.setenv("LBGPU_MP_RESIDENT", "grid")
    rho = np.where(NAT == 0, 1.0, 0.0)
    with Box(NAT, precision=precision) as box:
        box.mp_init(moments=(rho, [0.0 * rho] * 3), Db=0.01, ka=0.01 * math.e, kd=0.01)
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "20")
        with pytest.raises(LbgpuError) as e:
            box.mp_propagate(20)
        assert e.value.status == ERR_TIMEOUT


@pytest.mark.parametrize("at", [1, 2, 5, 30])
def test_charges(monkeypatch, at):
    nat = geo.cc(16, 16, 16)
    with Box(nat) as box:
        box.pnp_init(bjl=0.4, sigma=-1.0, lambda_D=4.0, D_plus=0.05, D_minus=0.05)
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", str(at + 1))
        with pytest.raises(LbgpuError) as e:
            box.sor()
        assert e.value.status == ERR_TIMEOUT


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
@pytest.mark.parametrize("wait", ["1", "20"])
def test_a_lost_tracer_state_stays_lost(monkeypatch, precision, wait):
    """Neither steps nor results of it until the state is set or formed anew."""
    monkeypatch.setenv("LBGPU_MP_RESIDENT", "grid")
    rho = np.where(NAT == 0, 1.0, 0.0)
    tr = dict(moments=(rho, [0.0 * rho] * 3), Db=0.01, ka=0.01 * math.e, kd=0.01)
    with Box(NAT, precision=precision) as box:
        box.mp_init(**tr)
        box.mp_propagate(5)
        state = box.mp_get()
        box.mp_propagate(20)
        want = box.mp_get()
        for again in (lambda: box.mp_set(*state, it_next=6), lambda: (box.mp_init(**tr), box.mp_propagate(5))):
            monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", wait)
            with pytest.raises(LbgpuError):
                box.mp_propagate(20)
            monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
            for call in (lambda: box.mp_propagate(3), box.mp_get, lambda: box.time_mp_steps(3)):
                with pytest.raises(LbgpuError) as e:
                    call()
                assert e.value.status == ERR_TIMEOUT
            again()
            box.mp_propagate(20)
            assert all(np.array_equal(x, y) for x, y in zip(box.mp_get(), want))


@pytest.mark.parametrize("wait", ["1", "12"])
@pytest.mark.parametrize("loop", [True, False])
def test_a_lost_charge_state_stays_lost(monkeypatch, wait, loop):
    nat = geo.cc(16, 16, 16)
    charges = dict(bjl=0.4, sigma=-1.0, lambda_D=4.0, D_plus=0.05, D_minus=0.05)
    with Box(nat) as box:
        box.pnp_init(**charges)
        state = box.pnp_get()
        box.sor()
        want = box.pnp_get()
        for again in (lambda: box.pnp_set(*state), lambda: box.pnp_init(**charges)):
            box.pnp_set(*state)
            monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", wait)
            with pytest.raises(LbgpuError):
                box.poisson_nernst_planck(max_outer=3) if loop else box.sor()
            monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
            for call in (box.pnp_get, box.sor, box.just_eq_smolu, box.poisson_residual, box.electrostatic_pot,
                         lambda: box.poisson_nernst_planck(max_outer=2)):
                with pytest.raises(LbgpuError) as e:
                    call()
                assert e.value.status == ERR_TIMEOUT
            with pytest.raises(LbgpuError):
                box.mp_init(moments=(np.where(nat == 0, 1.0, 0.0), [np.zeros(nat.shape)] * 3), Db=0.01, z=1.0, charged=True)
            again()
            box.sor()
            got = box.pnp_get()
            assert all(np.array_equal(x, y) for x, y in zip(got[:3], want[:3])) and got[3] == want[3]
