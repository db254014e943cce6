"""Result arrays in fresh and in used memory, aligned to nothing, below and above the size at which
their pages are made by several threads; and states built again and again over an older one of the
same context, against states of a fresh one (all bit for bit)."""
import ctypes as C

import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
@pytest.mark.parametrize("side", [5, 41, 71])
def test_flow_get_into_fresh_and_used_arrays(side, precision):
    nat = geo.cc(side, side, side)
    with Box(nat, f_ext=(1e-5, 0, 0), precision=precision) as box:
        box.flow_init()
        box.flow_steps(6)
        used = [np.ones(19 * nat.size + 3)[1:-2].reshape((19,) + nat.shape)] + [np.ones(nat.size + 1)[1:].reshape(nat.shape) for _ in range(4)]
        rc = box.L.lbgpu_flow_get(box.ctx, *(a.ctypes.data_as(C.POINTER(C.c_double)) for a in used))
        assert rc == 0
        box.flow_steps(2)
        n, rho, j = box.flow_get()
        with Box(nat, f_ext=(1e-5, 0, 0), precision=precision) as other:
            other.flow_init()
            other.flow_steps(6)
            m, rho6, j6 = other.flow_get()
    assert np.array_equal(used[0], m) and np.array_equal(used[1], rho6)
    assert all(np.array_equal(a, b) for a, b in zip(used[2:], j6))
    assert not np.array_equal(n, m)


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_tracer_states_over_older_ones(precision):
    nat = geo.slit(6, 7, 20)
    kinds = [dict(ka=0.03, kd=0.01), dict(), dict(ka=0.03, kd=0.01), dict(ka=0.05, kd=0.02)]

    def solve(box, kind):
        v0 = box.mp_init(Db=0.01, f_ext=(1e-5, 0, 0), **kind)
        vacf, _ = box.mp_propagate(40)
        return [v0, vacf, *box.mp_get()]

    def fresh():
        box = Box(nat, f_ext=(1e-5, 0, 0), precision=precision)
        box.flow_init()
        box.flow_steps(30)
        return box

    with fresh() as box:
        again = [solve(box, k) for k in kinds]
    for kind, got in zip(kinds, again):
        with fresh() as box:
            assert all(np.array_equal(a, b) for a, b in zip(solve(box, kind), got))


def test_charge_states_over_older_ones():
    nat = geo.slit(6, 6, 20)

    def solve(box, solver):
        box.pnp_init(sigma=-0.05, lambda_D=3.0, solver=solver, omega=1.8, tol=1e-5)
        box.poisson_nernst_planck(max_outer=3, check=False)
        return box.pnp_get()

    order = [0, 1, 0, 2, 1]
    with Box(nat) as box:
        again = [solve(box, s) for s in order]
    for s, got in zip(order, again):
        with Box(nat) as box:
            assert all(np.array_equal(a, b) for a, b in zip(solve(box, s), got))


def test_history_buffer_grows_and_is_cleared():
    nat = geo.slit(4, 4, 10)
    with Box(nat, f_ext=(1e-5, 0, 0)) as box:
        hists = []
        for cap in (20, 50, 200000, 10):
            box.flow_init()
            hist = np.full(cap, 7.0)
            steps = C.c_int(0)
            box.L.lbgpu_equilibration(box.ctx, 15, hist.ctypes.data_as(C.POINTER(C.c_double)), cap, C.byref(steps))
            hists.append(hist)
    assert all(np.array_equal(h[:10], hists[0][:10]) for h in hists)
    assert not hists[1][steps.value:].any() and not hists[2][steps.value:].any()


def test_batch_results_in_one_array_and_in_four():
    with Batch() as b:
        box = b.add(geo.cc(14, 14, 14), f_ext=(1e-5, 0, 0), tracer=dict(Db=0.01, ka=0.03, kd=0.01))
        b.steps(20)
        rho, j = b.moments(box)
        apart = [np.empty(rho.size + 2)[2:] for _ in range(4)]
        ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
        assert b.L.lbgpu_batch_moments(b.b, box, *(ptr(a) for a in apart)) == 0
        assert all(np.array_equal(a, x.ravel()) for a, x in zip(apart, (rho, *j)))
        b.mp_start(box)
        b.steps(10)
        P, A = b.mp_fields(box)
        apart = [np.empty(P.size + 2)[2:] for _ in range(2)]
        assert b.L.lbgpu_batch_mp_fields(b.b, box, ptr(apart[0]), ptr(apart[1])) == 0
        assert np.array_equal(apart[0], P.ravel()) and np.array_equal(apart[1], A.ravel())
        assert A.any() and P.any()
