"""The Poisson-Nernst-Planck loop of a small box in one launch against launches per step and a host
loop: Jacobi sweeps bit for bit (their operations are the same; both against the oracle too), sweep and
outer counts equal, ion densities to 1e-12 of their largest (the flux sums only decide; a node's update
is the same operations), at the edges of the resident form and of one-node-wide boxes."""
import numpy as np
import pytest

from laboetie_gb300 import Box, LbgpuError
from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import ERR_STEP_CAP, POISSON_JACOBI, POISSON_REFERENCE

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 1 << 10
CHARGES = dict(bjl=0.4, lambda_D=4.0, D_plus=0.05, D_minus=0.04)


def random_box(shape, seed):
    nat = (np.random.default_rng(seed).random(shape) < 0.35).astype(np.int8)
    nat.flat[0], nat.flat[-1] = 0, 1
    return nat


def run(monkeypatch, mode, nat, what, solver=POISSON_REFERENCE, **kw):
    monkeypatch.setenv("LBGPU_PNP_RESIDENT", mode)
    with Box(nat) as box:
        inter = box.interfacial()
        sigma = -0.01 * int(((nat == 1) & (inter == 1)).sum())
        box.pnp_init(sigma=sigma, solver=solver, **CHARGES, **kw)
        out = what(box)
        return out, box.pnp_get()


SHAPES = [(1, 1, 2), (1, 1, 64), (64, 1, 1), (3, 2, 5), (9, 8, 7), (31, 1, 17), (16, 16, 16), (33, 21, 19),
          (48, 48, 48), (64, 48, 38), (65, 48, 38)]   # 64*48*38 = 116736 = 152 * 768


@pytest.mark.parametrize("shape", SHAPES)
def test_sweeps_bit_identical(oracle_mod, monkeypatch, shape):
    nat = random_box(shape, sum(shape))

    def what(box):
        try:
            box.sor()
        except LbgpuError as e:
            assert e.status == ERR_STEP_CAP
    kw = dict(solver=POISSON_JACOBI, omega=1.4, tol=1e-5, max_iter=37)
    _, a = run(monkeypatch, "0", nat, what, **kw)
    _, b = run(monkeypatch, "1", nat, what, **kw)
    inter = oracle_mod.detect_interfacial(nat)
    sigma = -0.01 * int(((nat == 1) & (inter == 1)).sum())
    cp, cm, phi, an, _ = oracle_mod.charges_init(nat, inter, 0.4, sigma, 4.0)
    try:
        phi, *_ = oracle_mod.sor(nat, sigma, 0.4, cp, cm, phi, an, omega=1.4, tol=1e-5, maxiter=37)
        assert np.array_equal(a[2], phi)
    except oracle_mod.OracleError:
        pass
    assert np.array_equal(a[2], b[2]) and a[3] == b[3]


@pytest.mark.parametrize("bug", [True, False])
@pytest.mark.parametrize("shape", [(1, 1, 40), (20, 1, 1), (3, 2, 5), (9, 8, 7), (13, 1, 17), (24, 20, 22), (48, 48, 48)])
def test_outer_loop(monkeypatch, shape, bug):
    nat = geo.cc(48, 48, 48) if shape == (48, 48, 48) else random_box(shape, 3 + sum(shape))
    what = lambda box: box.poisson_nernst_planck(max_outer=12, check=False)
    oa, a = run(monkeypatch, "0", nat, what, np_loop_bug=bug)
    ob, b = run(monkeypatch, "1", nat, what, np_loop_bug=bug)
    assert oa == ob
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x - y).max() <= 1e-12 * np.abs(x).max()
    assert abs(a[3] - b[3]) <= 1e-12 * abs(a[3])


def test_continues_across_launches_and_to_equilibrium(monkeypatch):
    """A slit converges after a few thousand outer iterations (several launches), and a solve with a
    tolerance of zero runs to its cap (more sweeps than one launch runs)."""
    nat = geo.slit(2, 1, 24)
    what = lambda box: box.poisson_nernst_planck(max_outer=50000, check=False)
    oa, a = run(monkeypatch, "0", nat, what)
    ob, b = run(monkeypatch, "1", nat, what)
    assert oa[2] == ob[2] == 0 and oa[1] == ob[1] and abs(oa[0] - ob[0]) <= 1
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x - y).max() <= 1e-10 * np.abs(x).max()

    def capped(box):
        with pytest.raises(LbgpuError) as e:
            box.sor()
        assert e.value.status == ERR_STEP_CAP
    kw = dict(solver=POISSON_JACOBI, omega=1.2, tol=0.0, max_iter=9000)
    _, a = run(monkeypatch, "0", nat, capped, **kw)
    _, b = run(monkeypatch, "1", nat, capped, **kw)
    assert np.array_equal(a[2], b[2])


def test_wait_runs_out(monkeypatch):
    nat = geo.slit(4, 4, 64)
    monkeypatch.setenv("LBGPU_PNP_RESIDENT", "1")
    with Box(nat) as box:
        box.pnp_init(sigma=-0.3, **CHARGES)
        monkeypatch.setenv("LBGPU_TEST_GRID_WAIT", "1")
        with pytest.raises(LbgpuError) as e:
            box.sor()
        assert e.value.status == ERR_TIMEOUT
        monkeypatch.delenv("LBGPU_TEST_GRID_WAIT")
        box.pnp_init(sigma=-0.3, **CHARGES)
        assert box.sor() > 0
