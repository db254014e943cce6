"""The FP64 strict step from arbitrary states, bit for bit against the oracle's operators: its integer
sums and divisions at the edges of their range (populations of very different size at a node, zero,
negative, non-finite, tiny and huge ones; fluxes that vanish, exact quotients, |j| above rho) and the
forms of the collision by relaxation time (1; c1 a power of two; any)."""
import numpy as np
import pytest

from laboetie_gb300 import FP64, Box

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).reshape(19, 1, 1, 1)
SHAPE = (5, 6, 13)


def _state(kind, rng):
    n = W * (1.0 + 0.02 * rng.standard_normal((19,) + SHAPE))
    if kind == "spread":        # up to 2^9 between the populations of a node: across the range of 2^7
        n = n * 2.0 ** (9 * rng.random((19,) + SHAPE))
    elif kind == "dyadic":      # sums and many quotients exact, ties among the roundings
        n = rng.integers(1, 64, (19,) + SHAPE) * 2.0 ** -8
    elif kind == "symmetric":   # j = 0 exactly
        n = np.broadcast_to(W, (19,) + SHAPE) * (1.0 + 0.1 * rng.random(SHAPE))
    elif kind == "large_first":  # rho beyond 2^62 units: many populations of the largest binade
        n = np.ones((19,) + SHAPE) * (1.0 + 0.99 * rng.random((19,) + SHAPE))
    elif kind == "odd":
        flat = n.reshape(-1)
        at = rng.permutation(flat.size)[:90]
        flat[at] = np.resize([0.0, -0.0, -0.01, 5e-324, 1e-310, 1e-200, 3.0, 1e5, 1e200], 90)
    elif kind == "tiny":
        n = n * 2.0 ** -700
    elif kind == "huge":
        n = n * 2.0 ** 600
    elif kind == "nonfinite":
        flat = n.reshape(-1)
        flat[rng.permutation(flat.size)[:3]] = [np.inf, np.nan, -np.inf]
    return np.ascontiguousarray(n)


@pytest.mark.parametrize("tau,f", [(1.0, (1e-5, 0, 0)), (0.8, (1e-5, -2e-5, 3e-6)), (2 / 3, (0, 0, 1e-4)), (2.0, (0, 0.01, 0)),
                                   (1.3, (0, 0, 0)), (1e6, (1e-5, 0, 2e-5)), (1e6, (-0.9, 0, 0))])
@pytest.mark.parametrize("kind", ["near", "spread", "dyadic", "symmetric", "large_first", "odd", "tiny", "huge", "nonfinite"])
def test_steps_from_any_state(oracle_mod, kind, tau, f):
    rng = np.random.default_rng(31)
    nat = (rng.random(SHAPE) < 0.25).astype(np.int8)
    n0 = _state(kind, rng)
    n0[:, nat != 0] = 0.0
    rho0 = n0.sum(0)
    j0 = [0.1 * rho0 * rng.uniform(-1, 1, SHAPE) * (kind != "symmetric") for _ in range(3)]
    zero = [np.zeros(SHAPE)] * 3
    force = [np.where(nat == 0, v, 0.0) for v in f]
    fluid = nat == 0
    with np.errstate(all="ignore"):
        n = oracle_mod.bounce_back_stream(nat, oracle_mod.collide(nat, tau, n0, rho0, j0, zero))
        _, rho, j, _ = oracle_mod.moments(nat, n, zero, zero)
        n = oracle_mod.bounce_back_stream(nat, oracle_mod.collide(nat, tau, n, rho, j, force))
        _, rho, j, _ = oracle_mod.moments(nat, n, force, j)
        n = oracle_mod.bounce_back_stream(nat, oracle_mod.collide(nat, tau, n, rho, j, force))
        _, rho, j, _ = oracle_mod.moments(nat, n, force, j)
    with Box(nat, relaxation_time=tau, f_ext=f, precision=FP64) as box:
        box.flow_set(n0, rho0, j0)
        box.flow_steps(3)
        gn, grho, gj = box.flow_get()
    assert np.array_equal(gn[:, fluid], n[:, fluid], equal_nan=True)
    assert np.array_equal(grho[fluid], rho[fluid], equal_nan=True)
    if kind != "nonfinite":   # there the oracle's j has the NaN of 0 * inf, a term the device leaves out
        assert all(np.array_equal(a[fluid], b[fluid], equal_nan=True) for a, b in zip(gj, j))
