"""The FP32 reference loop's check: its l2err history against FP64 sums of the same states, and its
population tests on values around -w rho0 and on non-finite ones."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import ERR_NEGATIVE_POPULATION, ERR_NONFINITE

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (7, 1, 33), (16, 16, 16), (13, 17, 19)])
def test_history_is_that_of_fp64_sums(shape):
    """l2err(t) = max |j(t) - j(t-1)|: the j the library reports for the states are FP64 sums of the
    same FP32 deviations; two such sums differ by at most 20 rounding errors of the largest
    deviation (18 additions and the force), i.e. 20 * 2^-53 * max|d|."""
    nat = (np.random.default_rng(1).random(shape) < 0.2).astype(np.int8)
    nat.flat[0] = 0
    f = (3e-5, -1e-5, 2e-5)
    steps = 12
    js, hist, dmax = [], None, 0.0
    for k in range(3, steps + 1):
        with Box(nat, relaxation_time=0.8, f_ext=f, precision=FP32_DEV) as box:
            box.flow_init()
            _, hist, _ = box.equilibration(max_steps=k, hist_cap=steps, check=False)
            n, rho, j = box.flow_get()
        js.append(np.array(j))
        d = n - W[:, None, None, None] * (nat == 0)
        dmax = max(dmax, np.abs(d).max())
    want = [np.abs(b - a).max() for a, b in zip(js, js[1:])]
    assert np.abs(np.array(want) - hist[3:]).max() <= 2 * 20 * 2.0 ** -53 * max(dmax, 1e-30)


# (offset of one population from zero in float steps around -w rho0, or a value) -> status
@pytest.mark.parametrize("l,rho0", [(0, 1.0), (3, 1.0), (11, 0.7), (5, 123.456)])
@pytest.mark.parametrize("kind", ["below", "at", "above", "nan", "inf", "-inf"])
def test_population_tests(l, rho0, kind):
    nat = geo.slit(3, 4, 6)
    n = (W[:, None, None, None] * np.where(nat == 0, rho0, 0.0)).copy()
    x = -W[l] * rho0
    t = np.float32(x)
    if float(t) < x:
        t = np.nextafter(t, np.float32(np.inf))       # the smallest float not below -w rho0
    d = {"below": np.nextafter(t, np.float32(-np.inf)), "at": t, "above": np.nextafter(t, np.float32(np.inf)),
         "nan": np.float32(np.nan), "inf": np.float32(np.inf), "-inf": np.float32(-np.inf)}[kind]
    # the collision that precedes the first check spreads a non-finite value, and a call reports the
    # negative populations first
    want = {"below": ERR_NEGATIVE_POPULATION, "at": 0, "above": 0}.get(kind, ERR_NONFINITE)
    z, y, xx = 2, 1, 1
    n[l, z, y, xx] = float(d) + W[l] * rho0 if np.isfinite(d) else d
    rho, j = n.sum(0), [np.zeros(nat.shape)] * 3
    with Box(nat, rho0=rho0, relaxation_time=1e30, precision=FP32_DEV) as box:
        # tau 1e30: the collision leaves the populations as they are, so the check of the first
        # step sees the value where it streamed to
        box.flow_set(n, rho, j)
        _, _, rc = box.equilibration(max_steps=1, check=False)
    if want == ERR_NONFINITE:
        assert rc in (ERR_NONFINITE, ERR_NEGATIVE_POPULATION)
    else:
        assert rc & (ERR_NEGATIVE_POPULATION | ERR_NONFINITE) == want
