"""LBGPU_FP64_FUSED keeps the momentum of a box without walls or force: what a step adds to it is the
rounding of the populations to doubles and no drift of the fixed-point arithmetic.

Bound: a step rounds the 12 diagonal populations (near 1/36, last bit 2^-58) and 6 axis ones (near 1/18,
2^-57) of a node, each with a standard deviation of 0.29 of its last bit; a component of the flux takes 8
and 2 of them: 0.29 2^-58 (8 + 2 4)^1/2 = 1.2 2^-58 a node and step, the populations at rest included.  Six
standard deviations of the sum."""
import math
from fractions import Fraction

import numpy as np
import pytest

from laboetie_gb300 import FP64_FUSED, Box

pytestmark = pytest.mark.gpu

C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
              (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1),
              (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)])
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).reshape(19, 1, 1, 1)


def _flux(n):
    return [math.fsum(x for l in range(19) if C[l, d] for x in (C[l, d] * n[l]).ravel()) for d in range(3)]


@pytest.mark.parametrize("resident", ["0", None])
@pytest.mark.parametrize("tau", [0.8, 1.0, 0.62, 1.37])
def test_no_drift(monkeypatch, tau, resident):
    if resident is not None:
        monkeypatch.setenv("LBGPU_F64_RESIDENT", resident)
    shape, steps = (20, 22, 24), 240
    rng = np.random.default_rng(3)
    n0 = W * (1 + 1e-3 * rng.standard_normal((19,) + shape))
    with Box(np.zeros(shape, dtype=np.int8), relaxation_time=tau, precision=FP64_FUSED) as box:
        box.flow_set(n0, n0.sum(0), [np.zeros(shape)] * 3)
        box.flow_steps(1)
        a = _flux(box.flow_get()[0])
        box.flow_steps(steps)
        b = _flux(box.flow_get()[0])
    bound = 6 * 1.2 * 2.0 ** -58 * math.sqrt(np.prod(shape) * steps)
    assert all(abs(x - y) <= bound for x, y in zip(a, b)), [(x - y) / bound for x, y in zip(a, b)]


def test_no_loss_from_small_populations():
    """Populations some 2^-11 of their node's largest one, whose last bits lie below the fixed-point grid
    (unit 2^-59 for a largest one in [1, 2)), cost the node no mass beyond the share by which the rounded
    constants of the collision miss 1.  The mean over the nodes, in units: the rest population's rounding to
    a double (last bit 2^-52 = 128 units) has a standard deviation of 37 a node, and one unit for the share's
    own rounding."""
    shape, tau = (24, 30, 32), 50.0
    rng = np.random.default_rng(9)
    n0 = 1e-4 * rng.uniform(1, 2, (19,) + shape)
    n0[0] = rng.uniform(1.1, 1.2, shape)
    with Box(np.zeros(shape, dtype=np.int8), relaxation_time=tau, precision=FP64_FUSED) as box:
        box.flow_set(n0, n0.sum(0), [np.zeros(shape)] * 3)
        box.flow_steps(1)
        a = box.flow_get()[0]
        box.flow_steps(1)
        b = box.flow_get()[0]
    assert a[0].min() >= 1.0 and a[1:].max() < 2.0 ** -8
    c1, c2 = 1.0 - 1.0 / tau, 1.0 / tau
    share = 1 - Fraction(c1) - Fraction(c2 * (1 / 3)) - 6 * Fraction(c2 * (1 / 18)) - 12 * Fraction(c2 * (1 / 36))
    gained = math.fsum(np.concatenate([b.ravel(), -a.ravel()])) + float(share) * a.sum()
    units = gained / np.prod(shape) * 2.0 ** 59
    assert abs(units) <= 6 * 37 / math.sqrt(np.prod(shape)) + 1, units
