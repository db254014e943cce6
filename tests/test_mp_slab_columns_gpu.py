"""The staged FP32 tracer step at the edges of its tiles and chunks: two columns of y per thread (odd
and even last rows), chunks of 4 planes and fewer, halos that wrap; P and its adsorbed part have the
bits of the grid-stride step, VACF agrees to the rounding of FP32 sums (a thread adds up to lz terms
in sequence: lz 2^-24 of the sum of their magnitudes, itself below the value at t = 0)."""
import numpy as np
import pytest

from laboetie_gb300 import FP32_DEV, Box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ads", [dict(), dict(ka=0.02, kd=0.01)])
@pytest.mark.parametrize("shape", [(3, 8, 32), (4, 9, 33), (5, 10, 64), (7, 15, 34), (8, 16, 32), (9, 17, 63), (33, 11, 40)])
def test_columns_and_chunks(monkeypatch, shape, ads):
    rng = np.random.default_rng(23)
    nat = (rng.random(shape) < 0.35).astype(np.int8)
    rho = np.where(nat == 0, 1.0 + 1e-3 * rng.standard_normal(shape), 0.0)
    j = [np.where(nat == 0, 1e-3 * rng.standard_normal(shape), 0.0) for _ in range(3)]
    out = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("LBGPU_MP_SLAB", mode)
        with Box(nat, precision=FP32_DEV) as box:
            v0 = box.mp_init(moments=(rho, j), Db=0.01, **ads)
            vacf, _ = box.mp_propagate(21)
            out[mode] = (vacf, *box.mp_get())
    assert np.array_equal(out["1"][1], out["0"][1]) and np.array_equal(out["1"][2], out["0"][2])
    assert np.abs(out["1"][0] - out["0"][0]).max() <= shape[0] * 2.0 ** -24 * np.abs(v0).max()
