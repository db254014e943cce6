"""The work that a user has this library do, as cases that can be timed and checked.

Every case is one pass of a user's program through the package's public entry points (``Box``,
``Batch``), with sizes of the repository's own benchmark, tests and synthetic workloads:

* ``flow``: a flow solve from rest -- the reference's two-phase loop (``loop``) or fixed steps --
  and the density and flux it ends with;
* ``tracer``: the moment propagation of an (adsorbing) tracer in a box's flow state;
* ``pnp``: the Poisson-Nernst-Planck loop of charged solutes from the initial charges;
* ``operators``: one step of the Fortran loop left as it is, operator by operator on host arrays;
* ``batch_flow`` / ``batch_tracer``: many uneven boxes stepped together;
* ``serve``: a stream of requests through the continuous-batching server.

``exact`` restates the physics in torch in 64 bits, without this package's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from laboetie_gb300 import FP32_DEV, FP64, FP64_FUSED, Box
from laboetie_gb300 import geometry as geo
from laboetie_gb300 import workloads as wl
from laboetie_gb300.lbgpu import POISSON_REFERENCE, POISSON_SOR4, Batch

PRECISION = {"fp64": FP64, "fused": FP64_FUSED, "fp32": FP32_DEV}
TRACER_DB, TRACER_KD = 0.01, 0.01


# ------------------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest ordinary solve: a chromatography cell of the reference's tutorial in the
        # reference's arithmetic, to a step cap (default relaxation time 1)
        dict(name="cell_fp64_loop", kind="flow", geom="cell", lx=1, ly=50, lz=50, precision="fp64",
             tau=1.0, steps=400, loop=True),
        # the smallest box of the serving families, a narrow slit, FP32 fixed steps
        dict(name="slit_fp32_steps", kind="flow", geom="slit", lx=4, ly=4, lz=77, precision="fp32",
             tau=1.0, steps=1000, loop=False),
        # a ragged porous sample in the reference's arithmetic and loop
        dict(name="porous_fp64_loop", kind="flow", geom="porous", lx=97, ly=90, lz=101,
             precision="fp64", tau=0.8, steps=100, loop=True),
        # a porous box in the fused FP64 mode, fixed steps
        dict(name="porous_fused_steps", kind="flow", geom="porous", lx=128, ly=128, lz=128,
             precision="fused", tau=0.8, steps=120, loop=False),
        # touching spheres of odd side, the reference's loop in FP32
        dict(name="spheres_fp32_loop", kind="flow", geom="cc", lx=61, ly=61, lz=61,
             precision="fp32", tau=1.0, steps=400, loop=True),
        # the headline benchmark box, FP32 fixed steps: the largest flow
        dict(name="porous_fp32_steps", kind="flow", geom="porous", lx=192, ly=192, lz=192,
             precision="fp32", tau=0.8, steps=1000, loop=False),
        # an adsorbing tracer in the reference's arithmetic
        dict(name="tracer_fp64", kind="tracer", geom="porous", lx=64, ly=70, lz=75,
             precision="fp64", tau=0.8, steps=300, ads=True),
        # an adsorbing tracer in FP32 in a large porous box
        dict(name="tracer_fp32", kind="tracer", geom="porous", lx=160, ly=160, lz=160,
             precision="fp32", tau=0.8, steps=2000, ads=True),
        # charged touching spheres: a cold Poisson solve, then outer iterations
        dict(name="pnp_spheres", kind="pnp", geom="cc", lx=48, ly=48, lz=48, solver="reference",
             outer=60),
        # the reference's Fortran loop left as it is: one step on host arrays
        dict(name="operators_fp64", kind="operators", geom="cavity", lx=41, ly=41, lz=41, tau=1.0),
        # a parameter sweep of chromatography cells with modulated tubes among them, flow phase
        dict(name="batch_flow", kind="batch_flow", cells=256, tubes=16, steps=1000),
        # the same boxes in their tracer phase
        dict(name="batch_tracer", kind="batch_tracer", cells=256, tubes=16, steps=600),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, vmax, precision="fp64"):
    """geometry family and sides of one drawn box of at most vmax nodes (the fused mode is for
    three-dimensional media)."""
    geom = rng.choice(("porous", "porous", "cc", "cavity", "cylinder", "slit", "cell"))
    if precision == "fused" and geom != "cc":
        geom = "porous"
    v = _log(rng, 800, vmax)
    if geom == "cell":
        return dict(geom=geom, lx=1, ly=rng.randint(28, 70), lz=rng.randint(28, 70))
    if geom == "slit":
        return dict(geom=geom, lx=rng.randint(1, 8), ly=rng.randint(1, 8), lz=rng.randint(16, 128))
    if geom == "cylinder":
        n = max(10, min(96, int((v / 16) ** 0.5)))
        return dict(geom=geom, lx=n, ly=n, lz=rng.randint(8, 40))
    if geom in ("cc", "cavity"):
        n = max(9, int(v ** (1 / 3)))
        return dict(geom=geom, lx=n, ly=n, lz=n)
    n = max(12.0, v ** (1 / 3))
    a, b = rng.uniform(0.75, 1.2), rng.uniform(0.75, 1.1)
    return dict(geom="porous", lx=int(n * a), ly=int(n * b), lz=max(9, int(n / (a * b))))


def draw(rng):
    kind = rng.choice(("flow", "flow", "flow", "tracer", "tracer", "pnp", "operators", "batch_flow",
                       "batch_tracer", "serve"))
    if kind == "flow":
        precision = rng.choice(("fp64", "fused", "fp32", "fp32"))
        c = dict(kind=kind, precision=precision, tau=rng.choice((1.0, 1.0, 0.8, rng.uniform(0.55, 1.4))),
                 loop=rng.random() < 0.5, **_box(rng, 5e6 if precision == "fp32" else 1.2e6, precision))
        c["steps"] = int(max(40, min(800, (1.5e8 if precision == "fp32" else 4e7) / _nodes(c))))
        return c
    if kind == "tracer":
        precision = rng.choice(("fp64", "fused", "fp32", "fp32"))
        c = dict(kind=kind, precision=precision, tau=rng.choice((1.0, 0.8)), ads=rng.random() < 0.6,
                 **_box(rng, 3e6 if precision == "fp32" else 5e5, precision))
        c["steps"] = int(max(60, min(1000, (4e8 if precision == "fp32" else 1e8) / _nodes(c))))
        return c
    if kind == "pnp":
        b = dict(geom="slit", lx=rng.randint(1, 4), ly=rng.randint(1, 4), lz=rng.randint(20, 48))
        if rng.random() < 0.6:
            n = rng.randint(16, 48)
            b = dict(geom="cc", lx=n, ly=n, lz=n)
        return dict(kind=kind, solver=rng.choice(("reference", "reference", "sor")), outer=rng.randint(1, 60), **b)
    if kind == "operators":
        return dict(kind=kind, tau=rng.choice((1.0, 0.8)), **_box(rng, 1e5))
    if kind == "serve":
        return dict(kind=kind, stream=rng.randint(1, 10 ** 6), requests=rng.randint(4, 10), mp_steps=rng.randint(2, 12) * 100)
    return dict(kind=kind, cells=int(_log(rng, 16, 300)), tubes=int(_log(rng, 2, 20)),
                steps=2 * rng.randint(100, 300))


def _nodes(c):
    return c["lx"] * c["ly"] * c["lz"]


# --------------------------------------------------------------------------------- inputs

def _nature(c, seed):
    g, lx, ly, lz = c["geom"], c["lx"], c["ly"], c["lz"]
    if g == "cell":
        return geo.chromatography_cell(seed, ny=ly, nz=lz, radius=5.0 if min(ly, lz) >= 50 else 3.0)
    if g == "slit":
        return geo.slit(lx, ly, lz)
    if g == "cylinder":
        return wl.cylinder_r(lx, lz, lx / 2 - 2)
    if g == "cc":
        return geo.cc(lx, ly, lz)
    if g == "cavity":
        return geo.spherical_cavity(lx, ly, lz)
    L = max(lx, ly, lz)
    nat = geo.porous_spheres(L, 8.0 if L >= 48 else 3.0, 0.60, seed)
    return np.ascontiguousarray(nat[:lz, :ly, :lx])


def _force(c, seed):
    """f_ext of the solve: along z for the cells and cylinders, else along x, of the benchmark's size."""
    f = 1e-5 * float(np.random.default_rng(seed).uniform(0.3, 2.0))
    return (0.0, 0.0, f) if c["geom"] in ("cell", "cylinder") else (f, 0.0, 0.0)


def _tracer(ads, f):
    return dict(Db=TRACER_DB, ka=TRACER_KD * math.e if ads else 0.0, kd=TRACER_KD if ads else 0.0, f_ext=f)


def _batch_boxes(c, seed):
    """(nature, f_ext) per box: random cells; the tubes' lengths and order belong to the case."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(c["cells"])
    f = (0.0, 0.0, wl.FEXT * float(rng.uniform(0.3, 2.0)))
    boxes = [geo.chromatography_cell(seed=int(rng.integers(1 << 62)), ny=50, nz=50) for _ in range(c["cells"])]
    boxes += [geo.modulated_tube(int(sizes.integers(64, 257)), r_amp=float(rng.uniform(2.0, 4.0)))
              for _ in range(c["tubes"])]
    return [(nat, f) for nat in boxes]


def _stream(c, seed):
    """The case's request stream (families, sizes), with forces of the seed."""
    r = np.random.default_rng(seed)
    out = []
    for q in wl.serving_stream(c["stream"], c["requests"], 1e6, max_steps=2000, mp_steps=c["mp_steps"]):
        f = tuple(v * float(r.uniform(0.3, 2.0)) for v in q["f_ext"])
        out.append(dict(q, f_ext=f, tracer=dict(q["tracer"], f_ext=f), moments=True))
    return out


def _charges(c, seed, nat):
    r = np.random.default_rng(seed)
    inter = np.zeros(nat.shape, dtype=bool)
    for cx, cy, cz in C[1:]:
        inter |= np.roll(nat, (cz, cy, cx), axis=(0, 1, 2)) != nat
    n = int(((nat == 1) & inter).sum())
    return dict(bjl=0.4, sigma=-0.01 * n * float(r.uniform(0.8, 1.25)), lambda_D=4.0, D_plus=0.05, D_minus=0.05)


def _operator_arrays(c, seed, nat):
    r = np.random.default_rng(seed)
    rho = 1.0 + 0.02 * r.standard_normal(nat.shape)
    rho[nat == 1] = 0.0
    n = W[:, None, None, None] * rho * (1.0 + 0.01 * r.standard_normal((19,) + nat.shape))
    j = [np.where(nat == 0, 1e-3 * r.standard_normal(nat.shape), 0.0) for _ in range(3)]
    f = [np.where(nat == 0, v, 0.0) for v in _force(c, seed)]
    return n, rho, j, f


FLOW_BEFORE_TRACER = 100


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind in ("batch_flow", "batch_tracer"):
        b = Batch()
        s["ids"] = [b.add(nat, f_ext=f, tracer=_tracer(True, f)) for nat, f in _batch_boxes(c, seed)]
        s["batch"] = b
        if kind == "batch_tracer":
            b.steps(FLOW_BEFORE_TRACER)
            for i in s["ids"]:
                b.mp_start(i)
        return s
    if kind == "serve":
        s["requests"] = _stream(c, seed)
        s["batch"] = Batch()
        return s
    nat, f = _nature(c, seed), None
    if kind == "pnp":
        s["box"] = Box(nat)
        s["charges"] = _charges(c, seed, nat)
        return s
    f = _force(c, seed)
    s["box"] = Box(nat, relaxation_time=c["tau"], f_ext=f, precision=PRECISION[c.get("precision", "fp64")])
    if kind == "operators":
        s["arrays"] = _operator_arrays(c, seed, nat)
    if kind == "tracer":
        s["tracer"] = _tracer(c["ads"], f)
        s["box"].flow_init()
        s["box"].flow_steps(FLOW_BEFORE_TRACER)
        s["box"].sync()
    return s


# ------------------------------------------------------------------------------- one pass

def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "flow":
        box = s["box"]
        box.flow_init()
        hist = None
        if c["loop"]:
            hist = np.zeros(c["steps"])
            steps, h, _ = box.equilibration(max_steps=c["steps"], hist_cap=c["steps"], check=False)
            hist[:steps] = h
        else:
            box.flow_steps(c["steps"])
        _, rho, j = box.flow_get(populations=False)
        return [rho, *j, hist]
    if kind == "tracer":
        box = s["box"]
        v0 = box.mp_init(**s["tracer"])
        vacf, _ = box.mp_propagate(c["steps"])
        P, A = box.mp_get()
        return [_held(c, v0), _held(c, vacf), P, A]
    if kind == "pnp":
        box = s["box"]
        box.pnp_init(solver=POISSON_SOR4 if c["solver"] == "sor" else POISSON_REFERENCE, omega=1.8, tol=1e-5,
                     **s["charges"])
        outer, sweeps, _ = box.poisson_nernst_planck(max_outer=c["outer"], check=False)
        cp, cm, phi, _ = box.pnp_get()
        return [cp, cm, phi, outer, sweeps]
    if kind == "operators":
        box = s["box"]
        n, rho, j, f = s["arrays"]
        n = box.collide(n, rho, j, f)
        n = box.bounce_back_stream(n)
        _, rho, j, err = box.moments(n, f, j)
        return [n, rho, *j, err]
    b = s["batch"]
    if kind == "batch_flow":
        b.steps(c["steps"], check=True)
        out = [b.moments(i) for i in s["ids"]]
        return [_cat(o[0] for o in out)] + [_cat(o[1][d] for o in out) for d in range(3)]
    if kind == "batch_tracer":
        b.steps(c["steps"])
        v = [b.mp_get(i) for i in s["ids"]]
        f = [b.mp_fields(i) for i in s["ids"]]
        return [np.array([x[q] for x in v], dtype=np.float32) for q in range(3)] + [_cat(x[0] for x in f),
                                                                                   _cat(x[1] for x in f)]
    res = b.serve(s["requests"], du_tol=1e-7, check_every=100)
    out = [_cat(r["moments"][0] for r in res)] + [_cat(r["moments"][1][d] for r in res) for d in range(3)]
    return out + [np.array([r["vacf0"] for r in res], dtype=np.float32),
                  np.array([r["vacf_sum"] for r in res], dtype=np.float32),
                  np.array([r["steps"] for r in res])]


def _cat(arrays):
    return np.concatenate([a.ravel() for a in arrays])


def _held(c, v):
    """VACF values as they are held: sums of FP32 terms in an FP32 box."""
    return np.asarray(v, dtype=np.float32) if c["precision"] == "fp32" else np.asarray(v)


# ------------------------------------------------------------------------------- the work

FLUID = {"porous": 0.6, "cc": 0.32, "cavity": 0.5, "cylinder": 0.7, "slit": 0.95, "cell": 0.82}


def work(case):
    c, kind = case, case["kind"]
    if kind == "flow":
        nf, size = FLUID[c["geom"]] * _nodes(c), 4 if c["precision"] == "fp32" else 8
        return {"bytes": c["steps"] * nf * 38 * size + 32 * _nodes(c), "flops": c["steps"] * nf * 250}
    if kind == "tracer":
        nf = FLUID[c["geom"]] * _nodes(c)
        per = 40 if c["precision"] == "fp32" else 18 * 8 + 48 + 32
        return {"bytes": c["steps"] * nf * per + 48 * _nodes(c), "flops": c["steps"] * nf * 160}
    if kind == "pnp":
        sweeps = c["outer"] + (25 * c["lx"] if c["solver"] == "reference" else 2 * c["lx"])
        return {"bytes": (32 * sweeps + 200 * c["outer"]) * _nodes(c), "flops": 45 * sweeps * _nodes(c)}
    if kind == "operators":
        return {"bytes": (4 * 19 + 18) * 8 * _nodes(c), "flops": 350 * _nodes(c)}
    if kind == "serve":
        nf = 5e4 * c["requests"]
        return {"bytes": nf * (1000 * 152 + c["mp_steps"] * 40), "flops": nf * (1000 * 250 + c["mp_steps"] * 160)}
    nodes = 2050 * c["cells"] + 50000 * c["tubes"]
    per = (152, 250) if kind == "batch_flow" else (40, 160)
    return {"bytes": c["steps"] * nodes * per[0], "flops": c["steps"] * nodes * per[1]}


# ------------------------------------------------------------- the same physics in 64 bits

C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
     (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
     (0, -1, -1)]
INV = [C.index((-x, -y, -z)) for x, y, z in C]
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Lattice:
    """The D3Q19 lattice over the fluid nodes (or all nodes) of several boxes laid end to end."""

    def __init__(self, natures, all_nodes=False):
        d = _dev()
        self.shapes = [n.shape for n in natures]
        nat = torch.cat([torch.from_numpy(n.reshape(-1)).to(d) for n in natures])
        self.total = nat.numel()
        self.solid = nat != 0
        self.keep = torch.arange(self.total, device=d) if all_nodes else torch.nonzero(~self.solid).view(-1)
        self.n = self.keep.numel()
        place = torch.zeros(self.total, dtype=torch.int64, device=d)
        place[self.keep] = torch.arange(self.n, device=d)
        me = torch.arange(self.n, device=d)
        self.src, self.open = [], []   # node x - c_l, and whether it is of the node's nature
        for x, y, z in C:
            at, parts = 0, []
            for sh in self.shapes:
                k = sh[0] * sh[1] * sh[2]
                idx = torch.arange(at, at + k, device=d).view(sh)
                parts.append(torch.roll(idx, (z, y, x), (0, 1, 2)).reshape(-1))
                at += k
            s = torch.cat(parts)[self.keep]
            same = nat[s] == nat[self.keep]
            self.src.append(torch.where(same, place[s], me))
            self.open.append(same)
        self.interfacial = ~torch.stack(self.open).all(0)
        self.c = torch.tensor(C, dtype=torch.float64, device=d)
        self.w = torch.tensor(W, dtype=torch.float64, device=d)[:, None]

    def whole(self, v, last=None):
        """v over the kept nodes as an array over all nodes (zero on the others)."""
        out = torch.zeros((self.total,) + ((last,) if last else ()), dtype=torch.float64, device=v.device)
        out[self.keep] = v
        return out.cpu().numpy()

    def stream(self, f):
        out = torch.empty_like(f)
        for l in range(19):
            out[l] = torch.where(self.open[l], f[l][self.src[l]], f[INV[l]])
        return out

    def moments(self, f, F):
        return f.sum(0), self.c.T @ f + (F / 2 if F is not None else 0)

    def collide(self, f, rho, j, F, tau):
        u = j / rho
        cj, cu = self.c @ j, self.c @ u
        neq = self.w * (rho + 3 * cj + 4.5 * cj * cu - 1.5 * (j * u).sum(0))
        out = (1 - 1 / tau) * f + neq / tau
        if F is not None:
            cF = self.c @ F
            out += (1 - 1 / (2 * tau)) * self.w * (3 * (cF - (u * F).sum(0)) + 9 * cu * cF)
        return out


def _exact_flow(lat, F, tau, steps, loop, target=1e-10, force_from=2, rest_force=False):
    """Steps from rest.  F: (3, n).  loop: the reference's two-phase loop; else the force acts from
    the collision that starts step `force_from` (rest_force: and in the moments of the rest state)."""
    f = lat.w.expand(19, lat.n).clone()
    on_m = on_c = False
    jold = torch.zeros(3, lat.n, dtype=torch.float64, device=f.device)
    hist, without = [], False
    rho, j = lat.moments(f, F if rest_force else None)
    for t in range(1, steps + 1):
        if not loop:
            on_c = t >= force_from
        f = lat.stream(lat.collide(f, rho, j, F if on_c else None, tau))
        on_m = on_c
        rho, j = lat.moments(f, F if on_m else None)
        if loop:
            hist.append(float((j - jold).abs().max()))
            jold = j
            if hist[-1] <= target and t > 2:
                if without:
                    break
                without = on_c = True
    return rho, j, np.array(hist + [0.0] * (steps - len(hist))) if loop else None


def _exact_tracer(lat, box_of, nboxes, rho, j, f, steps, ads):
    """The moment propagation of a tracer with f its force (3, n): VACF(0), VACF of every step (per
    box), P and P_ads."""
    d = rho.device
    ka, kd = (TRACER_KD * math.e, TRACER_KD) if ads else (0.0, 0.0)
    inter = lat.interfacial if ads else torch.zeros_like(lat.interfacial)
    per_box = lambda v: torch.zeros(v.shape[0], nboxes, dtype=torch.float64, device=d).index_add_(1, box_of, v)
    one = torch.ones(1, lat.n, dtype=torch.float64, device=d)
    bw = (1.0 / (per_box(one) + (math.e if ads else 0.0) * per_box(one * inter)))[0][box_of]
    V = (j + f) / rho
    P = torch.zeros(3, lat.n, dtype=torch.float64, device=d)
    us, v0, frac, into = torch.zeros_like(P), torch.zeros_like(P), torch.ones_like(rho), []
    for l in range(1, 19):
        c, rest = lat.c[l][:, None], 6 * TRACER_DB * W[l]
        nb, op = lat.src[INV[l]], lat.open[INV[l]]      # x + c_l
        out = torch.where(op, 3 * W[l] * (c * V).sum(0) + rest, 0.0)
        spp = torch.where(op, -3 * W[l] * (c * V[:, nb]).sum(0) + rest, 0.0)
        frac = frac - out
        us += c * out
        v0 += c * c * out * bw
        P -= c * spp * bw
        into.append((nb, spp))
    A = torch.zeros_like(P)
    stay = torch.where(inter, frac - ka, frac)
    vacf = []
    for _ in range(steps):
        vacf.append(per_box(P * us))
        n = stay * P + torch.where(inter, kd * A, 0.0)
        for nb, spp in into:
            n += spp * P[:, nb]
        A = torch.where(inter, (1 - kd) * A + ka * P, A)
        P = n
    return per_box(v0), torch.stack(vacf), P, A


def _exact_pnp(nat, q, solver, outer_cap):
    """The Poisson-Nernst-Planck loop from the initial charges."""
    d, shape = _dev(), nat.shape
    fluid = torch.from_numpy(nat == 0).to(d)
    nb = lambda v, c: torch.roll(v, c, (2, 1, 0))                    # value at x - c
    inter = torch.zeros_like(fluid)
    for c in C[1:]:
        inter |= nb(fluid, c) != fluid
    w = W.tolist()
    rho0 = 1 / (4 * math.pi * q["bjl"] * q["lambda_D"] ** 2)
    n_int, n_fl = int((~fluid & inter).sum()), int(fluid.sum())
    ss = q["sigma"] / n_int if n_int else 0.0
    sf = -q["sigma"] / n_fl
    wall = torch.where(inter, 0.5 * ss, 0.0).to(torch.float64)
    cp = torch.where(fluid, 0.5 * rho0 + max(sf, 0.0), wall)
    cm = torch.where(fluid, 0.5 * rho0 + max(-sf, 0.0), -wall)
    fac = 4 * math.pi * q["bjl"] / 6
    anorm = fac * float((cp + cm).sum())
    phi = torch.zeros(shape, dtype=torch.float64, device=d)
    ax = [torch.arange(n, device=d) for n in shape]
    ring = lambda x, n: torch.zeros_like(x) if n == 1 else torch.where((x == n - 1) & (n % 2 == 1), 2, x % 2)
    size = lambda n: 1 if n == 1 else 2 + n % 2
    gz, gy, gx = (ring(a, n) for a, n in zip(ax, shape))
    ka, kb = (max(size(n), size(shape[0])) for n in (shape[2], shape[1]))
    colour = (gx[None, None] + gz[:, None, None]) % ka + ka * ((gy[None, :, None] + gz[:, None, None]) % kb)
    masks = [colour == k for k in range(ka * kb)]
    total, n, done = 0, 0, False
    line = torch.ones_like(fluid)   # the sites that start links, as the reference's loop bounds have it
    line[:-1] = False
    line[:, :-1] = False
    while not done and n < outer_cap:
        old = (phi, cp, cm)
        it = 0
        if solver == "sor":
            phi, keep = phi.clone(), float(phi.sum())
            while True:
                res = 0.0
                for m in masks:
                    r = fac * (cp - cm)
                    for l in range(1, 19):
                        r = r + w[l] * nb(phi, C[l])
                    res = res + (r - phi / 1.5).abs()[m].sum()
                    phi = torch.where(m, -0.8 * phi + 1.8 * 1.5 * r, phi)
                it += 1
                if float(res) <= 1e-5 * anorm:
                    break
            phi = phi - (float(phi.sum()) - keep) / phi.numel()
            total += it
        else:
            while True:
                star = fac * (cp - cm)
                for l in range(19):
                    star = star + w[l] * nb(phi, C[l])
                res = float((star - phi).abs().sum())
                phi = 1.4 * star - 0.4 * phi
                it += 1
                if res <= float(np.float32(1e-5)) * anorm:
                    break
            total += it - 1
        anorm = float(phi.abs().sum())
        for _ in range(10):
            fp, fm = torch.zeros_like(phi), torch.zeros_like(phi)
            for l in range(1, 19, 2):
                c, back = C[l], tuple(-v for v in C[l])
                delta = 1.0 if l < 7 else math.sqrt(2.0)
                on = line & fluid & nb(fluid, back)
                e = torch.exp(nb(phi, back) - phi)
                Jp = torch.where(on, 0.5 * (1 + 1 / e) * (nb(cp, back) * e - cp) * 0.1 * q["D_plus"] / delta, 0.0)
                Jm = torch.where(on, 0.5 * (1 + e) * (nb(cm, back) / e - cm) * 0.1 * q["D_minus"] / delta, 0.0)
                fp += Jp - nb(Jp, c)
                fm += Jm - nb(Jm, c)
            cp, cm = torch.where(fluid, cp + fp, cp), torch.where(fluid, cm + fm, cm)
            t = [float(v[fluid].square().sum()) ** 0.5 / n_fl / (0.05 * rho0 * D) / q["sigma"]
                 for v, D in ((fp, q["D_plus"]), (fm, q["D_minus"]))]
            if not sum(t) > float(np.float32(5e-6)):
                break
        ch = []
        for new, was in zip((phi, cp, cm), old):
            m = was.abs() > 1e-12
            ch.append(float(((new - was) / was)[m].abs().sum()) / max(1, int(m.sum())))
        done = all(v < 1e-12 for v in ch)
        n += 1
    return [cp.cpu().numpy(), cm.cpu().numpy(), phi.cpu().numpy(), None, None]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "serve":    # its step counts follow from convergence tests on FP32 velocities
        return None
    t64 = lambda v: torch.as_tensor(np.asarray(v, dtype=np.float64), device=_dev())
    if kind in ("batch_flow", "batch_tracer"):
        boxes = _batch_boxes(c, seed)
        lat = _Lattice([b[0] for b in boxes])
        F = t64(boxes[0][1])[:, None].expand(3, lat.n)
        steps = c["steps"] if kind == "batch_flow" else FLOW_BEFORE_TRACER
        rho, j, _ = _exact_flow(lat, F, 1.0, steps, False, force_from=1, rest_force=True)
        if kind == "batch_flow":
            return [lat.whole(rho)] + [lat.whole(j[d]) for d in range(3)]
        sizes = torch.tensor([b[0].size for b in boxes], device=_dev())
        box_of = torch.repeat_interleave(torch.arange(len(boxes), device=_dev()), sizes)[lat.keep]
        v0, vacf, P, A = _exact_tracer(lat, box_of, len(boxes), rho, j, F, c["steps"], True)
        flat = [lat.whole(x.T.contiguous(), 3).ravel() for x in (P, A)]
        return [v.T.cpu().numpy() for v in (v0, vacf.sum(0), vacf[-1])] + flat
    nat = _nature(c, seed)
    if kind == "pnp":
        return _exact_pnp(nat, _charges(c, seed, nat), c["solver"], c["outer"])
    if kind == "operators":
        n, rho, j, f = _operator_arrays(c, seed, nat)
        lat = _Lattice([nat], all_nodes=True)
        n, rho, j, F = (t64(v).reshape(*sh, -1) for v, sh in ((n, (19,)), (rho, ()), (j, (3,)), (f, (3,))))
        n = lat.stream(torch.where(lat.solid, n, lat.collide(n, rho, j, F, c["tau"])))
        rho, j2 = lat.moments(n, F)
        return [n.cpu().numpy().reshape((19,) + nat.shape)] + [x.cpu().numpy().reshape(nat.shape) for x in (rho, *j2)] + [
            float((j2 - j).abs().max())]
    lat = _Lattice([nat])
    f = t64(_force(c, seed))[:, None].expand(3, lat.n)
    if kind == "flow":
        rho, j, hist = _exact_flow(lat, f, c["tau"], c["steps"], c["loop"])
        out = [x.reshape(nat.shape) for x in (lat.whole(rho), *(lat.whole(j[d]) for d in range(3)))] + [hist]
        # zero but for rounding: across a slit or cylinder, and once a closed cavity has come to rest
        for d in {"slit": (1, 2), "cylinder": (0, 1), "cavity": (0, 1, 2)}.get(c["geom"], ()):
            out[1 + d] = None
        return out
    rho, j, _ = _exact_flow(lat, f, c["tau"], FLOW_BEFORE_TRACER, False)
    v0, vacf, P, A = _exact_tracer(lat, torch.zeros_like(lat.keep), 1, rho, j, f, c["steps"], c["ads"])
    return [v0[:, 0].cpu().numpy(), vacf[:, :, 0].cpu().numpy()] + [
        lat.whole(x.T.contiguous(), 3).reshape(nat.shape + (3,)) for x in (P, A)]
