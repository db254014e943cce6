"""j / rho of the FP64 strict collision where the quotient is no normal number: a density and a flux from
opposite ends of the exponent range, each of which the integer division takes by itself.  Against the
oracle's IEEE division: bit for bit where the result is finite, and not finite where it is not (infinity
or NaN: the oracle also adds the 0 * inf of velocity components that are 0)."""
import numpy as np
import pytest

from laboetie_gb300 import FP64, Box

pytestmark = pytest.mark.gpu

# the exponents between which the quotient is a normal number, and both sides of each line
EXPONENTS = [-900, -767, -501, -500, -499, -100, 0, 100, 499, 500, 501, 700, 767, 900]


@pytest.mark.parametrize("force", [0.0, 1.0, 2.0 ** -300])
def test_collide_at_both_ends_of_the_range(oracle_mod, force):
    rng = np.random.default_rng(5)
    k = len(EXPONENTS)
    shape = (3, k, k)
    nat = np.zeros(shape, dtype=np.int8)
    m = lambda: rng.uniform(1.0, 2.0, shape) * rng.choice([-1.0, 1.0], shape)   # noqa: E731
    rho = np.abs(m()) * 2.0 ** np.array(EXPONENTS, dtype=float)[None, None, :]
    j = [m() * 2.0 ** np.array(EXPONENTS, dtype=float)[None, :, None] for _ in range(3)]
    n = rng.uniform(0.5, 1.0, (19,) + shape)
    f = [np.full(shape, force * v) for v in (1.0, -0.5, 0.25)]
    with np.errstate(all="ignore"):
        want = oracle_mod.collide(nat, 1.3, n, rho, j, f)
    with Box(nat, relaxation_time=1.3, precision=FP64) as box:
        got = box.collide(n, rho, j, f)
    fine = np.isfinite(want)
    assert 0.2 < fine.mean() < 1.0
    assert np.array_equal(np.isfinite(got), fine)
    assert np.array_equal(got[fine], want[fine])
