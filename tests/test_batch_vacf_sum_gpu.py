"""The VACF of a batched box's node tiles is the sum of its nodes' FP32 terms as a single box forms it (exact
within a warp, FP64 beyond), late in the decay, where the terms cancel.  Bound: FP64 additions over the
warps and tiles, some 2^5 of them in a row, of 2^-53 of the terms' magnitude each: 2^-47 of it.  The
terms' magnitude: |P| times |u*|, the scattering's mean displacement, below lambda/2 = 6 Db for a fluid
almost at rest."""
import math

import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import Batch

pytestmark = pytest.mark.gpu

F = (0.0, 0.0, 1e-5)
TR = dict(Db=0.01, ka=0.01 * math.e, kd=0.01, f_ext=F)


@pytest.mark.parametrize("table", [True, False])
@pytest.mark.parametrize("nat", [geo.modulated_tube(48), geo.porous_spheres(40, 5.0, 0.6, 3)], ids=["tube", "porous"])
@pytest.mark.parametrize("steps", [2, 200])
def test_against_a_single_box(monkeypatch, nat, table, steps):
    monkeypatch.setenv("LBGPU_BATCH_SMEM", "0")
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "0")
    with Batch() as b:
        b.add(nat, f_ext=F, tracer=TR)
        need = b.info()["bytes"]
    with Batch(memory_budget=0 if table else need) as b:
        i = b.add(nat, f_ext=F, tracer=TR)
        b.steps(60)
        mom = b.moments(i)
        b.mp_start(i)
        b.steps(steps)
        got, (P, A) = b.mp_get(i), b.mp_fields(i)
    with Box(nat, f_ext=F, precision=FP32_DEV) as box:
        box.mp_init(moments=mom, **TR)
        box.mp_propagate(steps - 1)
        now = box.mp_get()[0]
        want, last = box.mp_propagate(1)[0][0], box.mp_get()
    assert np.array_equal(P, last[0]) and np.array_equal(A, last[1])
    bound = 2.0 ** -47 * 6 * TR["Db"] * np.abs(now).sum((0, 1, 2))
    assert (np.abs(got[2] - want) <= bound).all(), np.abs(got[2] - want) / bound
