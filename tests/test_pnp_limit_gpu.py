"""The stopping value of the solves within one call of the Poisson-Nernst-Planck loop is of SUM(ABS(phi))
in the reference's (storage) order, as it is from call to call: the tolerance at which a second solve takes
one sweep more is the same double for both, and so are the counts on either side of it."""
import numpy as np
import pytest

from laboetie_gb300 import Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import POISSON_JACOBI

pytestmark = pytest.mark.gpu


def charges(tol, sigma):
    return dict(bjl=0.4, sigma=sigma, lambda_D=4.0, D_plus=0.05, D_minus=0.05, solver=POISSON_JACOBI, omega=1.3, tol=tol)


def by_calls(box, tol, sigma):
    box.pnp_init(**charges(tol, sigma))
    n = box.sor()
    box.just_eq_smolu()
    return n + box.sor()


def by_loop(box, tol, sigma):
    box.pnp_init(**charges(tol, sigma))
    outer, sweeps, _ = box.poisson_nernst_planck(max_outer=2, check=False)
    assert outer == 2
    return sweeps


@pytest.mark.parametrize("side,sigma", [(12, -0.5), (17, -1.3), (24, -2.0)])
def test_same_threshold(side, sigma):
    with Box(geo.cc(side, side, side)) as box:
        lo, hi = 1e-4, 2e-4
        n_lo, n_hi = by_calls(box, lo, sigma), by_calls(box, hi, sigma)
        assert n_lo > n_hi
        while np.nextafter(lo, hi) < hi:
            mid = lo + (hi - lo) / 2
            if by_calls(box, mid, sigma) > n_hi:
                lo = mid
            else:
                hi = mid
        for k in range(-40, 41):
            tol = lo + k * np.spacing(lo)
            assert by_loop(box, tol, sigma) == by_calls(box, tol, sigma), k
