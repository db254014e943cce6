"""Calls that hand results back keep little device memory: at most 32 MiB a batch, counted into its budget,
and 12 MiB a tracer state; the results come all the same with no room left in the budget."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, FP64, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import Batch

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TR = dict(Db=0.01, ka=0.027, kd=0.01, f_ext=(0.0, 0.0, 1e-5))
SLACK = 8 << 20   # granularity of the driver's mappings


def held(call):
    """device bytes that a call keeps"""
    before = torch.cuda.mem_get_info()[0]
    out = call()
    return before - torch.cuda.mem_get_info()[0], out


def test_batch_workspace():
    nat = np.zeros((160, 160, 160), dtype=np.int8)
    with Batch() as b:
        i = b.add(nat, f_ext=(0.0, 0.0, 1e-5), tracer=TR)
        b.steps(2)
        kept, _ = held(lambda: b.moments(i))
        assert kept <= (32 << 20) + SLACK, kept >> 20
        b.mp_start(i)
        b.steps(2)
        kept, _ = held(lambda: b.mp_fields(i))
        assert kept <= (32 << 20) + SLACK, kept >> 20


@pytest.mark.parametrize("precision", [FP64, FP32_DEV])
def test_tracer_staging(precision):
    nat = np.zeros((180, 180, 180), dtype=np.int8)
    with Box(nat, precision=precision) as box:
        rho = np.ones(nat.shape)
        box.mp_init(moments=(rho, [np.zeros(nat.shape)] * 3), **TR)
        box.mp_propagate(2)
        kept, (P, A) = held(box.mp_get)
        assert kept <= (12 << 20) + SLACK, kept >> 20
        kept, _ = held(lambda: box.mp_set(P, A, it_next=3))
        assert kept <= SLACK, kept >> 20
        got = box.mp_get()
        assert np.array_equal(got[0], P) and np.array_equal(got[1], A)


def test_results_without_room_in_the_budget():
    """Large and small boxes, the budget just theirs: the workspace is not kept, nor any table."""
    boxes = [geo.modulated_tube(200), geo.cc(24, 24, 24), geo.modulated_tube(64)]

    def run(budget):
        with Batch(memory_budget=budget) as b:
            ids = [b.add(n, f_ext=(0.0, 0.0, 1e-5), tracer=TR) for n in boxes]
            used = b.info()["bytes"]
            b.steps(20)
            out = [b.moments(i) for i in ids]
            for i in ids:
                b.mp_start(i)
            b.steps(20)
            return used, out, [b.mp_fields(i) for i in ids], [b.mp_get(i) for i in ids]
    used, *want = run(0)
    _, *got = run(used)
    for a, b in zip(want[0], got[0]):
        assert np.array_equal(a[0], b[0]) and all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))
    for a, b in zip(want[1], got[1]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for a, b in zip(want[2], got[2]):
        assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))
