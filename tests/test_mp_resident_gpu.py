"""Tracer steps of small boxes in one launch (a cluster's shared memory, or a cooperative grid) against
one launch per step: P and P_ads bit for bit, VACF to 1e-12 of |VACF(0)| in FP64 (the node sum's order)
and to 1e-6 in FP32 boxes (a thread's FP32 sum of a few terms against exact sums: 2^-24 per term), in
every precision, at the edges of both forms, through interrupted runs, resumes and the convergence
test."""
import math

import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, FP64_FUSED, Box, LbgpuError
from laboetie_gb300 import geometry as geo

from test_flow_resident_gpu import box_with

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10
ADS = dict(Db=0.01, ka=0.01 * math.e, kd=0.01)


def moments(nat, seed):
    rng = np.random.default_rng(seed)
    fluid = nat == 0
    rho = np.where(fluid, 1.0 + 0.01 * rng.standard_normal(nat.shape), 0.0)
    return rho, [np.where(fluid, 1e-3 * rng.standard_normal(nat.shape), 0.0) for _ in range(3)]


def run(monkeypatch, mode, nat, precision, what, tracer):
    if mode is None:
        monkeypatch.delenv("LBGPU_MP_RESIDENT", raising=False)
    else:
        monkeypatch.setenv("LBGPU_MP_RESIDENT", mode)
    with Box(nat, precision=precision) as box:
        v0 = box.mp_init(moments=moments(nat, 5), f_ext=(1e-5, 0.0, 0.0), **tracer)
        out = what(box)
        P, A = box.mp_get()
    return v0, out, P, A


def same(a, b, precision):
    assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])
    tol = (1e-6 if precision == FP32_DEV else 1e-12) * np.abs(a[0]).max()
    for (va, ca), (vb, cb) in zip(a[1], b[1]):
        assert ca == cb and va.shape == vb.shape and np.abs(va - vb).max() <= tol


# FP32: cluster to 8192 nodes, grid to 77824; FP64: cluster to 2048, grid to 38912
@pytest.mark.parametrize("mode", [None, "grid", "cluster"])
@pytest.mark.parametrize("precision,nf", [(p, n) for p in (FP64, FP64_FUSED) for n in
                                          (1, 33, 513, 2048, 2049, 4096, 4097, 38912, 38913)] +
                         [(FP32_DEV, n) for n in (1, 33, 513, 8192, 8193, 40001, 77824, 77825)])
@pytest.mark.parametrize("ads", [True, False])
def test_steps(monkeypatch, precision, nf, mode, ads):
    if mode == "cluster" and nf > 9000:
        pytest.skip("beyond a cluster")
    nat = box_with(nf, nf + 1)

    def what(box):
        return [box.mp_propagate(1), box.mp_propagate(6), box.mp_propagate(17)]
    tr = ADS if ads else dict(Db=0.02)
    a = run(monkeypatch, "0", nat, precision, what, tr)
    same(a, run(monkeypatch, mode, nat, precision, what, tr), precision)


@pytest.mark.parametrize("mode", [None, "grid"])
@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_slab_and_grid_stride_agree_with_it(monkeypatch, precision, mode):
    nat = geo.porous_spheres(40, 5.0, 0.6, 3)   # wide enough for the slab step
    what = lambda box: [box.mp_propagate(30)]
    b = run(monkeypatch, mode, nat, precision, what, ADS)
    a = run(monkeypatch, "0", nat, precision, what, ADS)
    monkeypatch.setenv("LBGPU_MP_SLAB", "0")
    c = run(monkeypatch, mode, nat, precision, what, ADS)
    same(a, b, precision)
    same(c, b, precision)


@pytest.mark.parametrize("mode", [None, "grid"])
@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_convergence_ends_the_run_at_its_step(monkeypatch, precision, mode):
    """A closed cavity at rest: VACF decays until |VACF| < min(Db/(2 N), 1e-12); both forms stop at
    the same step (FP32: where an FP32 VACF first falls below it) with the P of that step."""
    nat = geo.spherical_cavity(9, 9, 9)
    rho = np.where(nat == 0, 1.0, 0.0)
    z = [np.zeros(nat.shape)] * 3

    def go(m):
        monkeypatch.setenv("LBGPU_MP_RESIDENT", m)
        with Box(nat, precision=precision) as box:
            v0 = box.mp_init(moments=(rho, z), Db=0.05)
            v, conv = box.mp_propagate(20000)
            P, A = box.mp_get()
            more, conv2 = box.mp_propagate(3)
        return v0, v, conv, P, more, conv2
    a, b = go("0"), go(mode or "1")
    assert a[2] == b[2]
    if precision == FP64:
        assert b[2] and 10 < len(b[1]) < 20000 and abs(len(a[1]) - len(b[1])) <= 1
    if len(a[1]) == len(b[1]):
        assert np.array_equal(a[3], b[3])
    assert a[4].shape == b[4].shape and a[5] == b[5]


def test_resume(monkeypatch):
    nat = box_with(3000, 4)
    for precision in (FP64, FP32_DEV):
        monkeypatch.delenv("LBGPU_MP_RESIDENT", raising=False)
        with Box(nat, precision=precision) as box:
            box.mp_init(moments=moments(nat, 1), **ADS)
            box.mp_propagate(7)
            P, A = box.mp_get()
            v, _ = box.mp_propagate(9)
            end = box.mp_get()
        with Box(nat, precision=precision) as box:
            box.mp_init(moments=moments(nat, 1), **ADS)
            box.mp_set(P, A, it_next=8)
            w, _ = box.mp_propagate(9)
            got = box.mp_get()
        assert np.array_equal(v, w) and np.array_equal(end[0], got[0]) and np.array_equal(end[1], got[1])


def test_wait_runs_out(monkeypatch):
    monkeypatch.setenv("LBGPU_MP_RESIDENT", "grid")
    nat = geo.slit(4, 4, 64)
    for precision in (FP64, FP32_DEV):
        with Box(nat, precision=precision) as box:
            box.mp_init(moments=moments(nat, 2), **ADS)
            monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
            with pytest.raises(LbgpuError) as e:
                box.mp_propagate(20)
            assert e.value.status == ERR_TIMEOUT
            monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
            box.mp_init(moments=moments(nat, 2), **ADS)
            assert len(box.mp_propagate(20)[0]) == 20
