"""The FP32 reference loop's check launch where a block takes several groups of 256 nodes: boxes whose
fluid nodes exactly fill one group per block (456 x 256), one node fewer and more, and many, with the
largest flux change in the first, a middle and the last group; its l2err against FP64 sums of the same
states, and a negative population found in any group."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, Box
from laboetie_gb300.lbgpu import ERR_NEGATIVE_POPULATION

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def _nature(fluid):
    nat = np.zeros((57, 32, 131), dtype=np.int8)
    nat.flat[fluid:] = 1
    return nat


@pytest.mark.parametrize("fluid", [456 * 256 - 1, 456 * 256, 456 * 256 + 1, 57 * 32 * 131])
@pytest.mark.parametrize("where", [0.0, 0.5, 1.0])
def test_largest_change_in_any_group(fluid, where):
    """As test_flow_fp32_check_gpu: two FP64 sums of the same deviations differ by at most 20 rounding
    errors of the largest one."""
    nat = _nature(fluid)
    rng = np.random.default_rng(4)
    n = W[:, None, None, None] * (1 + 1e-4 * rng.standard_normal((19,) + nat.shape)) * (nat == 0)
    hot = int(where * (fluid - 1))
    n.reshape(19, -1)[1, hot] += 0.02
    rho = n.sum(0)
    js, hist = [], None
    for k in (3, 4):
        with Box(nat, relaxation_time=0.9, f_ext=(1e-5, 0, 0), precision=FP32_DEV) as box:
            box.flow_set(n, rho, [np.zeros(nat.shape)] * 3)
            _, hist, _ = box.equilibration(max_steps=k, hist_cap=4, check=False)
            m, _, j = box.flow_get()
        js.append(np.array(j))
        dmax = np.abs(m - W[:, None, None, None] * (nat == 0)).max()
    want = np.abs(js[1] - js[0]).max()
    assert abs(want - hist[3]) <= 2 * 20 * 2.0 ** -53 * dmax


@pytest.mark.parametrize("where", [0.0, 0.37, 1.0])
def test_negative_population_in_any_group(where):
    nat = _nature(57 * 32 * 131)
    n = np.repeat(W, nat.size).reshape((19,) + nat.shape).copy()
    n.reshape(19, -1)[4, int(where * (nat.size - 1))] = -0.01
    with Box(nat, relaxation_time=1e30, precision=FP32_DEV) as box:
        box.flow_set(n, n.sum(0), [np.zeros(nat.shape)] * 3)
        _, _, rc = box.equilibration(max_steps=1, check=False)
    assert rc & ERR_NEGATIVE_POPULATION
