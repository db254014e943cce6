"""Boxes stepped by one launch for many steps (a cluster's shared memory, or a cooperative grid) against
one launch per step: the same populations, moments, l2err history and exit step, bit for bit, at the
edges of both forms, for fixed steps and for the reference loop with its force switch, exits and caps."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, Box, LbgpuError
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import ERR_NEGATIVE_POPULATION, ERR_STEP_CAP

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10


def box_with(nf, seed):
    """A ragged random box with exactly nf fluid nodes."""
    rng = np.random.default_rng(seed)
    n = int(np.ceil(nf * 1.2)) + 2
    lx = max(1, int(round(n ** (1 / 3) * rng.uniform(0.7, 1.3))))
    ly = max(1, int(round((n / lx) ** 0.5 * rng.uniform(0.8, 1.2))))
    lz = -(-n // (lx * ly))
    nat = np.ones(lx * ly * lz, dtype=np.int8)
    nat[rng.permutation(nat.size)[:nf]] = 0
    return nat.reshape(lz, ly, lx)


def run(monkeypatch, mode, nat, what, **kw):
    if mode is None:
        monkeypatch.delenv("LBGPU_AA_RESIDENT", raising=False)
    else:
        monkeypatch.setenv("LBGPU_AA_RESIDENT", mode)
    with Box(nat, precision=FP32_DEV, **kw) as box:
        out = what(box)
        n, rho, j = box.flow_get()
    return out, n, rho, j


def same(a, b):
    (oa, na, ra, ja), (ob, nb, rb, jb) = a, b
    assert np.array_equal(na, nb) and np.array_equal(ra, rb) and all(np.array_equal(x, y) for x, y in zip(ja, jb))
    if oa is not None:
        assert oa[0] == ob[0] and np.array_equal(oa[1], ob[1]) and oa[2] == ob[2]


# cluster of 1..16 blocks up to 8192 nodes, one block per SM up to 77824, then launch per step
SIZES = [1, 32, 33, 65, 512, 513, 2560, 2561, 8191, 8192, 8193, 40000, 77824, 77825]


@pytest.mark.parametrize("nf", SIZES)
@pytest.mark.parametrize("mode", [None, "grid", "cluster"])
def test_fixed_steps(monkeypatch, nf, mode):
    nat = box_with(nf, nf)

    def what(box):
        box.flow_init()
        box.flow_steps(9)
        box.flow_steps(3, force_on=False)
        box.flow_steps(16, force_on=False)
        box.flow_get(populations=False)
        box.flow_steps(11)
    kw = dict(relaxation_time=0.8, f_ext=(2e-5, -1e-5, 3e-6))
    same(run(monkeypatch, "0", nat, what, **kw), run(monkeypatch, mode, nat, what, **kw))


@pytest.mark.parametrize("nf", SIZES)
@pytest.mark.parametrize("mode", [None, "grid", "cluster"])
def test_reference_loop_to_a_cap(monkeypatch, nf, mode):
    nat = box_with(nf, nf + 7)

    def what(box):
        box.flow_init()
        box.flow_steps(1, force_on=False)   # the loop starts in the other phase
        r = box.equilibration(max_steps=15, hist_cap=15, check=False)
        box.flow_steps(10)
        return r
    kw = dict(relaxation_time=1.0, f_ext=(0.0, 1e-5, 0.0))
    a, b = run(monkeypatch, "0", nat, what, **kw), run(monkeypatch, mode, nat, what, **kw)
    same(a, b)
    assert b[0][2] == (ERR_STEP_CAP if b[0][0] == 15 else 0)   # a few nodes come to rest before


@pytest.mark.parametrize("mode", [None, "grid", "cluster"])
@pytest.mark.parametrize("cap", [0, 4, 3])
def test_reference_loop_switch_and_exit(monkeypatch, mode, cap):
    """From a perturbed state: the first convergence (force on) is met on the way, and without a cap
    the second one ends the loop; caps at and just before the switch."""
    nat = geo.slit(3, 4, 20)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    rng = np.random.default_rng(2)
    n = w[:, None, None, None] * (1 + 1e-3 * rng.standard_normal((19,) + nat.shape)) * (nat == 0)
    rho, j = n.sum(0), [np.zeros(nat.shape)] * 3

    def what(box):
        box.flow_set(n, rho, j)
        r = box.equilibration(max_steps=cap or 20000, hist_cap=20000, check=False)
        box.flow_steps(8)
        return r
    kw = dict(relaxation_time=0.9, f_ext=(1e-4, 0.0, 0.0), target_error=3e-5)
    a, b = run(monkeypatch, "0", nat, what, **kw), run(monkeypatch, mode, nat, what, **kw)
    same(a, b)
    if not cap:
        assert b[0][2] == 0 and b[0][0] > 10


@pytest.mark.parametrize("mode", [None, "grid", "cluster"])
def test_reference_loop_negative_population(monkeypatch, mode):
    nat = geo.slit(4, 4, 12)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    n = (w[:, None, None, None] * (nat == 0)).copy()
    n[5, 6, 2, 2] = -0.2
    rho, j = n.sum(0), [np.zeros(nat.shape)] * 3

    def what(box):
        box.flow_set(n, rho, j)
        return box.equilibration(max_steps=50, hist_cap=50, check=False)
    kw = dict(relaxation_time=1.7, f_ext=(1e-5, 0.0, 0.0))
    a, b = run(monkeypatch, "0", nat, what, **kw), run(monkeypatch, mode, nat, what, **kw)
    same(a, b)
    assert b[0][2] == ERR_NEGATIVE_POPULATION


def test_wait_runs_out(monkeypatch):
    """The grid waits for a block it does not have: every wait ends at its limit, the call reports it
    and the context stays usable."""
    monkeypatch.setenv("LBGPU_AA_RESIDENT", "grid")
    nat = geo.slit(4, 4, 64)
    with Box(nat, precision=FP32_DEV, f_ext=(1e-5, 0.0, 0.0)) as box:
        box.flow_init()
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
        _, _, rc = box.equilibration(max_steps=20, check=False)
        assert rc == ERR_TIMEOUT
        box.flow_init()
        box.flow_steps(20)
        with pytest.raises(LbgpuError) as e:
            box.sync()
        assert e.value.status == ERR_TIMEOUT
        monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
        box.flow_init()
        box.flow_steps(20)
        box.sync()
        got = box.flow_get()
    monkeypatch.setenv("LBGPU_AA_RESIDENT", "0")
    with Box(nat, precision=FP32_DEV, f_ext=(1e-5, 0.0, 0.0)) as box:
        box.flow_init()
        box.flow_steps(20)
        want = box.flow_get()
    assert np.array_equal(got[0], want[0])
