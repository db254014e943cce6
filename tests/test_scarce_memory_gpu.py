"""Calls on a device with little memory left: what they did before states kept their buffers for the next
one, and results were converted on the device, they still do."""
import gc

import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import POISSON_JACOBI, Batch

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TR = dict(Db=0.01, f_ext=(0.0, 0.0, 1e-5))
ADS = dict(ka=0.027, kd=0.01, **TR)
NAT = np.zeros((96, 96, 96), dtype=np.int8)
MOMENTS = (np.ones(NAT.shape), [np.full(NAT.shape, v) for v in (1e-3, 0.0, -2e-3)])


@pytest.fixture
def leave():
    """leave(bytes): takes device memory until about that much is free; leave(None): gives it back."""
    held = []

    def take(free):
        if free is None:
            held.clear()
            gc.collect()
            torch.cuda.empty_cache()
            return
        torch.cuda.synchronize()
        for _ in range(64):   # in pieces of whole 2 MiB pages
            more = (torch.cuda.mem_get_info()[0] - free) >> 21 << 21
            if more <= 0:
                break
            try:
                held.append(torch.empty(more, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                try:
                    held.append(torch.empty(more // 2 >> 21 << 21 or 1 << 21, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
    yield take
    take(None)


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_a_smaller_state_over_a_larger_one(leave, precision):
    """28 MB of moments to upload, 10 MB free, and an older state with 28 MB (FP32) or 42 MB (FP64) that the
    new one does not need."""
    with Box(NAT, precision=precision) as box:
        box.mp_init(moments=MOMENTS, **TR)
        box.mp_propagate(2)
        want = box.mp_get()
    with Box(NAT, precision=precision) as box:
        box.mp_init(moments=MOMENTS, **ADS)
        leave(10 << 20)
        box.mp_init(moments=MOMENTS, **TR)
        leave(None)
        box.mp_propagate(2)
        got = box.mp_get()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_fields_with_little_room(leave, precision):
    """6 MB free: less than the staging of the box's fields (12 MiB) takes."""
    with Box(NAT, precision=precision) as box:
        box.mp_init(moments=MOMENTS, **ADS)
        box.mp_propagate(3)
        leave(6 << 20)
        got = box.mp_get()
        box.mp_set(*got, it_next=4)
        leave(None)
        want = box.mp_get()
        assert all(np.array_equal(a, b) for a, b in zip(got, want)) and np.abs(got[0]).max() > 0


def test_batch_fields_with_little_room(leave):
    with Batch() as b:
        ids = [b.add(NAT[:64], f_ext=(0.0, 0.0, 1e-5), tracer=ADS), b.add(NAT, f_ext=(0.0, 0.0, 1e-5), tracer=ADS)]
        b.steps(4)
        for i in ids:
            b.mp_start(i)
        b.steps(4)
        leave(6 << 20)
        got = [b.mp_fields(i) for i in ids]
        leave(None)
        want = [b.mp_fields(i) for i in ids]
    for g, w in zip(got, want):
        assert all(np.array_equal(x, y) for x, y in zip(g, w)) and np.abs(g[0]).max() > 0


@pytest.mark.parametrize("precision,side", [(FP64, 40), (FP32_DEV, 60)])
def test_many_steps_per_launch_without_room(leave, monkeypatch, precision, side):
    """Room for the state of a box, and not for the workspace (16 MiB and one more P) of its many-step
    launches: one launch per step."""
    nat = (np.random.default_rng(4).random((side, side, side)) < 0.65).astype(np.int8)

    def run(box):
        box.mp_init(**ADS)
        leave(None)
        box.mp_propagate(7)
        return box.mp_get()
    out = []
    for free in (None, "less"):
        with Box(nat, precision=precision, f_ext=(1e-5, 0.0, 0.0)) as box:
            box.flow_init()
            box.flow_steps(5)
            box.sync()
            if free:
                leave(need - (10 << 20))
            before = torch.cuda.mem_get_info()[0]
            out.append(run(box))
            if not free:
                box.mp_release()
                box.mp_init(**ADS)
                need = before - torch.cuda.mem_get_info()[0]
    want, got = out
    assert all(np.array_equal(a, b) for a, b in zip(got, want)) and np.abs(got[0]).max() > 0


def test_charges_without_room_for_the_right_hand_side(leave):
    """17 MB of it at 128^3, with 10 MB less free than the state takes with it: the same sweeps."""
    nat = geo.cc(128, 128, 128)
    charges = dict(bjl=0.4, sigma=-20.0, lambda_D=4.0, D_plus=0.05, D_minus=0.05, solver=POISSON_JACOBI, omega=1.2, tol=1e-5)
    out = []
    for free in (None, "less"):
        with Box(nat, precision=FP32_DEV) as box:
            if free:
                leave(need - (10 << 20))
            before = torch.cuda.mem_get_info()[0]
            box.pnp_init(**charges)
            need = before - torch.cuda.mem_get_info()[0]
            leave(None)
            out.append((box.sor(), box.pnp_get()))
    (n, want), (m, got) = out
    assert n == m > 2 and want[3] == got[3]
    assert all(np.array_equal(a, b) for a, b in zip(got[:3], want[:3])) and np.abs(got[2]).max() > 0
