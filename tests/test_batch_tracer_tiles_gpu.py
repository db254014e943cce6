"""The tiled boxes' tracer step with and without the probability table, and in slab tiles: P and P_ads
bit for bit; VACF bit for bit between the two node-tile forms (the same sums) and to 1e-6 of |VACF(0)|
against slab tiles (FP32 terms grouped differently, 2^-24 per addition); tables given back to a box that
needs the room."""
import math

import numpy as np
import pytest

from laboetie_gb300 import geometry as geo
from laboetie_gb300.lbgpu import Batch

pytestmark = pytest.mark.gpu

TR = dict(Db=0.01, ka=0.01 * math.e, kd=0.01, f_ext=(0.0, 0.0, 1e-5))


def ragged(shape, seed, solid=0.4):
    nat = (np.random.default_rng(seed).random(shape) < solid).astype(np.int8)
    nat.flat[0] = 0
    return nat


def exact_count(shape, nf, seed):
    nat = np.ones(int(np.prod(shape)), dtype=np.int8)
    nat[np.random.default_rng(seed).permutation(nat.size)[:nf]] = 0
    return nat.reshape(shape)


BOXES = [ragged((33, 29, 37), 1), geo.modulated_tube(48), exact_count((20, 20, 20), 4096, 2),
         exact_count((20, 20, 20), 4097, 3), ragged((60, 61, 1), 4), ragged((9, 8, 64), 5, 0.0), geo.cc(41, 41, 41)]


def run(boxes, budget=0, steps=(2, 30), extra=None):
    with Batch(memory_budget=budget) as b:
        ids = [b.add(n, f_ext=(0.0, 0.0, 1e-5), tracer=TR) for n in boxes]
        b.steps(20)
        for i in ids:
            b.mp_start(i)
        b.steps(steps[0])
        if extra is not None:
            b.add(extra, f_ext=(0.0, 0.0, 1e-5))
        b.steps(steps[1])
        out = [(b.mp_get(i), b.mp_fields(i)) for i in ids]
        return out, b.info()["bytes"]


def same(a, b, exact):
    for (va, fa), (vb, fb) in zip(a, b):
        assert np.array_equal(fa[0], fb[0]) and np.array_equal(fa[1], fb[1])
        for x, y in zip(va[:3], vb[:3]):
            if exact:
                assert np.array_equal(x, y)
            else:
                assert np.abs(x - y).max() <= 1e-6 * max(np.abs(va[0]).max(), np.abs(x).max())
        assert va[3] == vb[3]


def test_table_and_slab_tiles(monkeypatch):
    monkeypatch.setenv("LBGPU_BATCH_SMEM", "0")
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "0")
    table, used = run(BOXES)
    plain, _ = run(BOXES, budget=used)          # no room for any table
    some, _ = run(BOXES, budget=used + 4096 * 72 + 300)   # room for one
    same(table, plain, True)
    same(table, some, True)
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "1")
    slab, _ = run(BOXES)
    same(table, slab, False)
    monkeypatch.delenv("LBGPU_BATCH_SLAB")
    default, _ = run(BOXES)
    same(table, default, False)


def test_tables_make_room_for_a_box(monkeypatch):
    monkeypatch.setenv("LBGPU_BATCH_SMEM", "0")
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "0")
    extra = ragged((24, 25, 26), 9)
    with Batch() as b:
        b.add(extra, f_ext=(0.0, 0.0, 1e-5))
        need = b.info()["bytes"]
    want, used = run(BOXES, extra=extra)
    got, _ = run(BOXES, budget=used, extra=extra)      # tables fill the rest until the box comes
    same(want, got, True)
    assert used > need


def test_slab_tiles_of_a_dense_box(monkeypatch):
    """96^3 all fluid: large and dense enough for slab tiles; the node tiles give the same P."""
    nat = geo.bulk(96, 96, 96)
    a, _ = run([nat], steps=(2, 6))
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "0")
    b, _ = run([nat], steps=(2, 6))
    same(a, b, False)


def test_a_pore_gone_nan_leaves_the_others_alone(monkeypatch):
    """Two pores without a connection, side by side in x, so that lanes of one warp hold nodes of both: the
    force makes the wide one's flow unstable and its tracer NaN; the narrow one's stays what it is without a
    table."""
    monkeypatch.setenv("LBGPU_BATCH_SMEM", "0")
    monkeypatch.setenv("LBGPU_BATCH_SLAB", "0")
    nat = np.ones((32, 16, 36), dtype=np.int8)
    nat[:, :, 1] = 0
    nat[:, :, 3:34] = 0
    nat[::8, ::6, 18] = 1   # obstacles: no laminar flow
    out = []
    for budget in (0, None):
        with Batch(memory_budget=used if budget is None else budget) as b:   # None: no room for the table
            i = b.add(nat, f_ext=(0.0, 0.0, 2e-2), tracer=TR)
            used = b.info()["bytes"]
            b.steps(4000)
            b.mp_start(i)
            b.steps(20)
            out.append(b.mp_fields(i))
    for table, plain in zip(*out):
        assert np.isnan(plain[:, :, 3]).any() and np.isfinite(plain[:, :, 1]).all()
        assert np.array_equal(table[:, :, 1], plain[:, :, 1])


@pytest.mark.parametrize("nat,slab", [(geo.porous_spheres(64, 8.0, 0.60, 1), True), (geo.porous_spheres(48, 8.0, 0.60, 1), False),
                                      (geo.cc(64, 64, 64), False), (geo.slit(32, 32, 64), False)],
                         ids=["porous64", "porous48", "spheres64", "slit32"])
def test_tiles_by_default(monkeypatch, nat, slab):
    """The form a box takes shows in the grouping of its VACF sums: half the nodes of its slab tiles fluid,
    and 64 of them at least, for slab tiles."""
    out = {}
    for mode in ("0", "1", None):
        if mode is None:
            monkeypatch.delenv("LBGPU_BATCH_SLAB")
        else:
            monkeypatch.setenv("LBGPU_BATCH_SLAB", mode)
        out[mode] = run([nat], steps=(2, 40))[0]
    assert not np.array_equal(out["0"][0][0][1], out["1"][0][0][1])
    same(out[None], out["1" if slab else "0"], True)
