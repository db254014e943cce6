"""A tracer whose P has left the finite numbers: the steps of many per launch give the VACF and the P that
one launch per step gives -- an infinite term makes the sum infinite, infinities of both signs NaN."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, Box

from test_flow_resident_gpu import box_with

pytestmark = pytest.mark.gpu


def run(monkeypatch, mode, precision, nat, values):
    """VACF and P of eight steps from non-finite values in three calls, and P of five more from finite ones."""
    monkeypatch.setenv("LBGPU_MP_RESIDENT", mode)
    fluid = np.argwhere(nat == 0)
    rho = np.where(nat == 0, 1.0, 0.0)
    j = [np.where(nat == 0, v, 0.0) for v in (1e-3, 2e-3, -3e-3)]
    with Box(nat, precision=precision) as box:
        box.mp_init(moments=(rho, j), Db=0.02)
        good, A = box.mp_get()
        bad = good.copy()
        for q, v in zip(fluid[::37], values):
            bad[tuple(q)] = v
        box.mp_propagate(4)
        box.mp_set(bad, A, it_next=1)
        vacf = np.concatenate([box.mp_propagate(n)[0] for n in (1, 3, 4)])
        P = box.mp_get()[0]
        box.mp_set(good, A, it_next=1)
        assert len(box.mp_propagate(5)[0]) == 5
        return vacf, P, box.mp_get()[0]


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
@pytest.mark.parametrize("nf", [900, 9000])
@pytest.mark.parametrize("values", [(np.inf,), (-np.inf, -np.inf), (np.inf, -np.inf), (np.nan,)])
def test_same_as_one_launch_per_step(monkeypatch, precision, nf, values):
    nat = box_with(nf, 3)
    want, got = (run(monkeypatch, m, precision, nat, values) for m in ("0", "1"))
    assert len(want[0]) == 8 and not np.isfinite(want[0]).any()
    for w, g in zip(want, got):
        assert np.array_equal(g, w, equal_nan=True)
    assert np.isfinite(got[2]).all()
