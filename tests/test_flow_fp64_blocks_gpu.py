"""The FP64 strict step at the edges of its launch shapes and of its exact-product forms: bit-identical
to the oracle for boxes around the block-size thresholds (608 and 9728 warps of fluid nodes), in the
relaxation-time-1 form and the general one, with every force mask; and the population checks on the
bits of special values."""
import numpy as np
import pytest

from laboetie_gb300 import FP64, Box
from laboetie_gb300.lbgpu import ERR_NEGATIVE_POPULATION, ERR_NONFINITE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau,f_ext", [(1.0, (1e-5, 0.0, 0.0)), (0.8, (0.0, 0.0, 2e-5)), (1.0, (1e-5, -2e-5, 3e-6)),
                                       (1.3, (0.0, 1e-5, 0.0)), (1.0, (0.0, 0.0, 0.0))])
@pytest.mark.parametrize("shape,solid", [((1, 1, 31), 0), ((1, 3, 11), 1), ((38, 32, 16), 0), ((38, 32, 16), 32),
                                         ((39, 32, 16), 479), ((76, 64, 64), 0), ((77, 64, 64), 4095)])
def test_loop_bit_identical(oracle_mod, shape, solid, tau, f_ext):
    if solid and shape[0] > 50 and f_ext[1]:
        pytest.skip("the largest boxes once per form")
    nat = np.zeros(shape, dtype=np.int8)
    nat.flat[np.random.default_rng(3).permutation(nat.size)[:solid]] = 1
    steps = 7
    ref = oracle_mod.equilibration(nat, tau=tau, f_ext=f_ext, max_steps=steps, check=False, nthreads=8)
    with Box(nat, relaxation_time=tau, f_ext=f_ext, precision=FP64) as box:
        box.flow_init()
        n_steps, hist, rc = box.equilibration(max_steps=steps, hist_cap=steps, check=False)
        n, rho, j = box.flow_get()
    assert n_steps == ref["steps"] and np.array_equal(hist, ref["l2err"])
    assert np.array_equal(rho, ref["rho"]) and all(np.array_equal(a, b) for a, b in zip(j, ref["j"]))
    fluid = nat == 0
    assert np.array_equal(n[:, fluid], ref["n"][:, fluid])


# value of one population -> status of the first step (-0 and the smallest denormal are fine)
@pytest.mark.parametrize("value,bits", [(-0.0, 0), (5e-324, 0), (-5e-324, ERR_NEGATIVE_POPULATION),
                                        (-1e-3, ERR_NEGATIVE_POPULATION), (np.inf, ERR_NONFINITE),
                                        (-np.inf, ERR_NEGATIVE_POPULATION | ERR_NONFINITE),
                                        (np.nan, ERR_NONFINITE), (-np.nan, ERR_NONFINITE)])
def test_population_checks(value, bits):
    nat = np.zeros((4, 5, 6), dtype=np.int8)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    n = np.repeat(w, nat.size).reshape((19,) + nat.shape).copy()
    n[7, 2, 3, 4] = value
    with Box(nat) as box:
        rc, *_ = box.moments(n, [np.zeros(nat.shape)] * 3, [np.zeros(nat.shape)] * 3)
    assert rc & (ERR_NEGATIVE_POPULATION | ERR_NONFINITE) == bits
