"""One step of LBGPU_FP64_FUSED against the collision in extended precision, at the edges of its
fixed-point form: populations of very different size at one node, |j| and the force around and beyond
its range, negative and tiny populations (FP64 form), relaxation times down to 1/2.

Bounds, with S the sum of |n| at a node and u = |j/rho|.  Fixed point (populations >= 0, u < 1/40,
|F| < S/400; the largest population is then at least S/19 and its binade S/38): one rounding to double
(2^-53 S), the rounded constants' share of the mass (up to 2^-52 S, rest population) and a few units of 2^-60 of the
binade.  FP64: sums of 19 terms (18 roundings) in rho, j and, divided by rho, in u, which enter with
weights of at most 1 (c2 <= 2): 64 2^-53 (S + |F|)(1 + u + |F/rho|)^2 max(1, S/|rho|)."""
import numpy as np
import pytest

from laboetie_gb300 import FP64_FUSED, Box

pytestmark = pytest.mark.gpu

LD = np.longdouble
C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
              (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1),
              (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)])
W = np.array([LD(1) / 3] + [LD(1) / 18] * 6 + [LD(1) / 36] * 12)


def _collided(n, rho, j, F, tau):
    u = [a / rho for a in j]
    ju = sum(a * b for a, b in zip(j, u))
    uF = sum(a * b for a, b in zip(u, F))
    out = np.empty_like(n)
    for l, c in enumerate(C):
        cj, cu, cF = (sum(int(c[d]) * v[d] for d in range(3)) for v in (j, u, F))
        q = W[l] * (rho + 3 * cj + LD(4.5) * cj * cu - LD(1.5) * ju)
        out[l] = n[l] + (q - n[l]) / tau + (1 - 1 / (2 * tau)) * W[l] * (3 * (cF - uF) + 9 * cu * cF)
    return out


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -900, 2.0 ** 960])
@pytest.mark.parametrize("tau,f", [(1.0, (1e-5, 0, 0)), (0.5, (0, 0, 0)), (0.8, (3e-3, -1e-300, 2e-4)),
                                   (1.7, (0, 0.3, -0.2)), (50.0, (0, 0, 0.06))])
@pytest.mark.parametrize("spread,speed", [(0.0, 0.02), (30.0, 0.02), (3.0, 0.3), (70.0, 1.5)])
def test_one_step(spread, speed, tau, f, scale):
    rng = np.random.default_rng(5)
    shape = (6, 8, 11)
    nat = np.zeros(shape, dtype=np.int8)
    rho0 = scale * 2.0 ** (spread * rng.uniform(-0.5, 0.5, shape))
    j0 = [rho0 * speed * rng.uniform(-1, 1, shape) * rng.integers(0, 2, shape) for _ in range(3)]
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).reshape(19, 1, 1, 1)
    F = tuple(float(scale * v) for v in f)
    states = []   # the populations that each of three steps streams in
    with Box(nat, relaxation_time=tau, f_ext=F, precision=FP64_FUSED) as box:
        box.flow_set(w * rho0, rho0, j0)
        for _ in range(3):
            box.flow_steps(1)
            states.append(box.flow_get()[0].astype(LD))
    for step in range(2):   # the step that switches the force on has no F/2 in j, later ones do
        _check(states[step], states[step + 1], 0.5 * step, [LD(v) for v in F], LD(tau))


def _check(n1, n2, half, F, tau):
    rho = n1.sum(0)
    j = [sum(int(C[l, d]) * n1[l] for l in range(19)) + F[d] * half for d in range(3)]
    want = _collided(n1, rho, j, F, tau)
    S, Fm = np.abs(n1).sum(0), max(abs(v) for v in F)
    u = sum(np.abs(v) for v in j) / np.abs(rho)
    fixed = (n1 >= 0).all(0) & (u < LD(1) / 40) & (Fm < S / 400) & (S > LD(2) ** -880)
    eps = LD(2) ** -53
    tol = np.where(fixed, 3 * eps * S, 64 * eps * (S + Fm) * (1 + u + Fm / np.abs(rho)) ** 2 * np.maximum(1, S / np.abs(rho)))
    for l, c in enumerate(C):
        err = np.abs(np.roll(n2[l], tuple(-c[::-1]), (0, 1, 2)) - want[l]) / tol   # at the node it left
        assert err.max() <= 1, (l, float(err.max()), float(err[fixed].max(initial=0)))
