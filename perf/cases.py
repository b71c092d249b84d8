"""Work that users of this library have it do, through its public entry points: matrix-free
and dense solves of sphere microstructures, the host-buffer pipelines, stress fields, batches
of realisations (linear and quadratic eigenstrain, spheres and ellipsoids), the bounded cube
and one training step of the learned preconditioner.

Inputs come from a seed alone (the library's own microstructure generators, host only).
`exact` restates the sphere path in FP64 with torch alone: outside a sphere the potentials
of a polynomial eigenstrain are finite sums of derivatives of r and 1/r, inside they are
polynomials.
"""
import ctypes
import functools
import itertools
import math

import numpy as np
import torch

import ibemproject_gb300 as g
from ibemproject_gb300 import batch as B
from ibemproject_gb300 import cases as C

SIG = (0.0, 0.0, 0.0, 0.0, 0.0, 1.0)
E0, NU0, NU1 = 70e9, 0.3, 0.2
PRECOND = {"block_jacobi": 0, "learned": 1, "neumann": 2}
FORM = {"fp64": 0, "mixed": 1, "bj": 2}


def listed():
    return [
        # one small microstructure: the call that a parameter scan or an optimiser repeats
        dict(name="solve-64", kind="solve", num=64, vf=0.15, contrast=5.714, precond="learned"),
        # the benchmark's microstructure through the host-buffer call: solution and stresses on a grid
        dict(name="host-2000", kind="host", num=2000, vf=0.15, contrast=5.714, precond="learned", grid=64),
        # a representative volume of production size, packed densely
        dict(name="solve-20000", kind="solve", num=20000, vf=0.25, contrast=5.714, precond="learned"),
        # many realisations of different sizes, volume fractions and contrasts, and their effective moduli
        dict(name="batch-linear", kind="batch", layout=24, nseg=24, lo=50, hi=300, precond="learned"),
        # the same with quadratic eigenstrain
        dict(name="batch-quadratic", kind="batch", layout=60, nseg=12, lo=50, hi=300, precond="block_jacobi"),
        # stresses of a known solution on a ragged grid in the default precision
        dict(name="field-fp64", kind="field", num=700, vf=0.2, layout=24, form="fp64", nx=41, ny=37, nz=29),
        # assembly and plain FP64 LU of one microstructure: the check that a user makes of the other forms
        dict(name="dense-fp64", kind="dense", num=300, vf=0.15, layout=24, form="fp64"),
        # the mixed-precision dense form at quadratic eigenstrain
        dict(name="dense-mixed", kind="dense", num=280, vf=0.2, layout=60, form="mixed"),
        # the bounded cube of the configurations (600 boundary elements, 64 spheres, 78 unknowns each), default form
        dict(name="cube-fp64", kind="cube", n_face=10, num=64, layout=78, form="fp64", grid=32),
        # a smaller bounded case in the mixed form
        dict(name="cube-mixed", kind="cube", n_face=7, num=21, layout=24, form="mixed", grid=19),
        # realisations with ellipsoids: assembled and solved with block-Jacobi GMRES
        dict(name="batch-ellipsoids", kind="ell_batch", nseg=6, lo=50, hi=300),
        # one training step of the learned preconditioner: loss, gradient, AdamW
        dict(name="train-step", kind="train", num=1500, nrhs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "host", "batch", "batch", "field", "dense", "dense", "cube", "ell_batch", "train"])
    vf, contrast = round(rng.uniform(0.1, 0.25), 3), round(rng.uniform(2.0, 20.0), 3)
    if kind == "solve":
        return dict(kind=kind, num=_log_int(rng, 20, 16000), vf=vf, contrast=contrast, precond=rng.choice(sorted(PRECOND)))
    if kind == "host":
        return dict(kind=kind, num=_log_int(rng, 50, 2000), vf=vf, contrast=contrast, precond=rng.choice(sorted(PRECOND)),
                    grid=_log_int(rng, 7, 64))
    if kind == "batch":
        layout = rng.choice([24, 60])
        lo = _log_int(rng, 10, 100)
        return dict(kind=kind, layout=layout, nseg=_log_int(rng, 2, 24 if layout == 24 else 12), lo=lo,
                    hi=lo + _log_int(rng, 10, 200),
                    precond=rng.choice(sorted(PRECOND)) if layout == 24 else "block_jacobi")
    if kind == "field":
        return dict(kind=kind, num=_log_int(rng, 5, 700), vf=vf, layout=rng.choice([24, 60, 78]),
                    form=rng.choice(["fp64", "mixed"]), nx=rng.randint(9, 41), ny=rng.randint(9, 41), nz=rng.randint(5, 31))
    if kind == "dense":
        layout = rng.choice([24, 60, 78])
        form = rng.choice(["fp64", "mixed", "bj"])
        return dict(kind=kind, num=_log_int(rng, 3, (7200 if form == "fp64" else 16800) // layout), vf=vf, layout=layout,
                    form=form)
    if kind == "cube":
        return dict(kind=kind, n_face=rng.randint(3, 9), num=_log_int(rng, 2, 60), layout=rng.choice([24, 60, 78]),
                    form=rng.choice(["fp64", "mixed"]), grid=rng.randint(5, 31))
    if kind == "ell_batch":
        lo = _log_int(rng, 10, 100)
        return dict(kind=kind, nseg=rng.randint(1, 5), lo=lo, hi=lo + _log_int(rng, 10, 150))
    return dict(kind=kind, num=_log_int(rng, 100, 1500), nrhs=rng.randint(1, 4))


# --------------------------------------------------------------------------- inputs
def _sphere_case(num, vf, contrast, seed, grid=0, r0=0.012):
    return C.generated_case(num, r0, vf, seed=seed, method="mc", grid=grid, E0=E0, nu0=NU0, E1=E0 * contrast, nu1=NU1)


def _side(c):
    return float(c.title.split("=")[1])


def _sizes(case, seed):
    """Realisation sizes spread evenly over [lo, hi]: another seed gives other microstructures of the same cost."""
    return [int(n) for n in np.linspace(case["lo"], case["hi"], case["nseg"]).round()]


def _realisations(case, seed):
    rng = np.random.default_rng(seed)
    return [_sphere_case(n, float(rng.uniform(0.1, 0.25)), float(rng.uniform(2, 20)), int(rng.integers(1 << 30)), r0=0.008)
            for n in _sizes(case, seed)]


def _network(seed):
    """Network weights as training leaves them: every edge weight near that of the Neumann series."""
    gen = torch.Generator().manual_seed(seed)
    h, out = 64, []
    for fan_in, fan_out in [(10, h)] + [(2 * h + 7, h), (2 * h, h)] * 3 + [(2 * h + 7, h), (h, 2)]:
        s = (1 if fan_out == h else 0.1) / math.sqrt(fan_in)
        out += [(torch.rand(fan_in * fan_out, generator=gen) * 2 - 1) * s, torch.full((fan_out,), 0.0 if fan_out == h else 0.9)]
    return torch.cat(out)


def _graph(case, seed):
    """Inputs of a training step: 16 nearest neighbours of random centres, their features, projections of four-digit pairs."""
    num, nrhs = case["num"], case["nrhs"]
    gen = torch.Generator().manual_seed(seed)
    side = (num / 0.15 * 4.19) ** (1 / 3)
    x = torch.rand(num, 3, generator=gen, dtype=torch.float64) * side
    a = 0.8 + 0.4 * torch.rand(num, generator=gen, dtype=torch.float64)
    d = torch.cdist(x, x) + torch.eye(num) * 1e9
    nbr = d.topk(16, largest=False).indices
    off = (x[:, None] - x[nbr]) / a[:, None, None]
    dist = off.norm(dim=2, keepdim=True).clamp_min(2.0)
    ratio = (a[nbr] / a[:, None])[..., None]
    ef = torch.cat([off, dist, ratio, dist - 1 - ratio, (2 / dist) ** 3], 2)
    xn = torch.cat([torch.ones(num, 3), torch.tensor([[1.0, 0, 0, 0, 0.57, NU0, NU1]]).expand(num, 7)], 1)
    z = torch.randn(nrhs, num, 24, generator=gen) * 0.05 / math.sqrt(nrhs * num)
    u = torch.randn(nrhs, num * 16, 2, 24, generator=gen) * 0.01 / math.sqrt(nrhs * num)
    params = _network(seed)
    m = torch.randn(params.numel(), generator=gen) * 1e-3
    v = torch.rand(params.numel(), generator=gen) * 1e-6 + 1e-8
    return dict(nbr=nbr.to(torch.int32).contiguous(), xn=xn.float(), ef=ef.float(), z=z, u=u, params=params, m=m, v=v)


def _field_inputs(case, seed):
    c = _sphere_case(case["num"], case["vf"], 5.714, seed)
    rng = np.random.default_rng(seed)
    scale = np.repeat([1.0, 0.3, 0.1], [6, 18, case["layout"] - 24])[:case["layout"]]
    a = c.radius[:, None]
    order = np.repeat([0, 1, 2], [6, 18, case["layout"] - 24])[None, :]
    e = (np.r_[[1.0, 0, 0, 1.0, 0, -3.0], np.zeros(case["layout"] - 6)] + 0.3 * rng.standard_normal((c.num, case["layout"]))) * scale
    return c, e / a ** order * 1e-11


def _ellipsoids(case, seed):
    rng = np.random.default_rng(seed)
    return [C.ellipsoid_case(n, a1=0.008, vf=float(rng.uniform(0.1, 0.25)), seed=int(rng.integers(1 << 30)),
                             E1=E0 * float(rng.uniform(2, 20)), method="mc") for n in _sizes(case, seed)]


def _cube(case, seed):
    """The bounded cube with spheres of a radius that leaves room for `num` of them."""
    r = min(0.05, 0.19 / max(1, case["num"]) ** (1 / 3))
    return C.bounded_cube_case(n_face=case["n_face"], num=case["num"], radius=r, grid=case["grid"], seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        cs = ([_sphere_case(case["num"], case["vf"], case["contrast"], seed)] if kind == "solve" else _realisations(case, seed))
        return dict(case=case, bt=B.DeviceBatch(cs, layout=case.get("layout", 24)), vol=np.array([_side(c) ** 3 for c in cs]),
                    params=_network(seed).cuda())
    if kind == "host":
        c = _sphere_case(case["num"], case["vf"], case["contrast"], seed, grid=case["grid"])
        return dict(case=case, c=c, params=_network(seed).numpy())
    if kind == "field":
        c, e = _field_inputs(case, seed)
        dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(case=case, c=c, cen=dev(c.centers), rad=dev(c.radius), e=dev(e),
                    out=torch.empty((n, 6), dtype=torch.float64, device="cuda"))
    if kind in ("dense", "ell_batch"):
        cs = [_sphere_case(case["num"], case["vf"], 5.714, seed)] if kind == "dense" else _ellipsoids(case, seed)
        return dict(case=case, bt=B.DeviceBatch(cs, layout=case.get("layout", 24)), vol=np.array([_side(c) ** 3 for c in cs]))
    if kind == "cube":
        return dict(case=case, c=_cube(case, seed))
    s = {k: v.cuda() for k, v in _graph(case, seed).items()}
    s.update(case=case, nrhs=case["nrhs"])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("solve", "batch"):
        bt = state["bt"]
        x, _ = B.solve(bt, B.farfield_rhs(bt, SIG), PRECOND[case["precond"]], params=state["params"])
        e, strain = B.effective_modulus(bt, x, SIG, volume=state["vol"])
        return dict(x=x, e_eff=e, strain=strain)
    if kind == "host":
        x, s, _ = g.run_host_mf(state["c"], PRECOND[case["precond"]], state["params"])
        return dict(x=x, stress=s)
    if kind == "field":
        c, out = state["c"], state["out"]
        side, dp = _side(c), ctypes.POINTER(ctypes.c_double)
        lo, hi, sig = (np.ascontiguousarray(v, dtype=np.float64) for v in (np.zeros(3), np.full(3, side), SIG))
        n = (ctypes.c_int * 3)(case["nx"], case["ny"], case["nz"])
        m = g.material(c.E0, c.nu0, c.E1, c.nu1)
        g.check(g.lib().ibem_e3d_field_grid(FORM[case["form"]], lo.ctypes.data_as(dp), hi.ctypes.data_as(dp), n,
                                            state["cen"].data_ptr(), state["rad"].data_ptr(), c.num, ctypes.byref(m),
                                            case["layout"], state["e"].data_ptr(), None, 0, None, 0, None, None,
                                            sig.ctypes.data_as(dp), out.data_ptr(), None))
        return dict(stress=out)
    if kind in ("dense", "ell_batch"):
        bt = state["bt"]
        x, _ = B.dense_batch_solve(bt, B.farfield_rhs(bt, SIG), FORM[case.get("form", "bj")], tol=1e-12)
        e, strain = B.effective_modulus(bt, x, SIG, volume=state["vol"])
        return dict(x=x, e_eff=e, strain=strain)
    if kind == "cube":
        x, s, _ = g.run_host(state["c"], layout=case["layout"], form=FORM[case["form"]])
        return dict(x=x, stress=s)
    loss, grad = B.loss_grad(state, case["num"], state["params"])
    p, m, v = state["params"].clone(), state["m"].clone(), state["v"].clone()
    B.adamw(p, grad, m, v, 20, lr=2e-3, weight_decay=1e-4)
    return dict(loss=loss, grad=grad, params=p, m=m, v=v)


def work(case):
    """Each input read once and each output written once; operations of the contracted pair sums (one strain and its
    derivatives per pair, per product), of the factorisations and of the boundary quadrature."""
    kind = case["kind"]
    pair = {24: 900, 60: 6000, 78: 6000}       # one pair of one product
    point = {24: 260, 60: 700, 78: 700}        # one (point, sphere) pair of a stress sum
    if kind in ("solve", "batch", "host"):
        sizes = _sizes(case, 0) if kind == "batch" else [case["num"]]
        layout, steps = case.get("layout", 24), 14
        pairs, n, pts = sum(k * k for k in sizes), sum(sizes), case.get("grid", 0) ** 3
        return {"bytes": 8.0 * (4 * n + layout * n + 9 * pts), "flops": float(pair[layout] * pairs * steps + point[24] * pts * n)}
    if kind == "field":
        pts = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8.0 * (case["num"] * (4 + case["layout"]) + 6 * pts), "flops": float(point[case["layout"]] * pts * case["num"])}
    if kind == "dense":
        n = case["num"] * case["layout"]
        return {"bytes": 8.0 * (4 * case["num"] + 2 * n), "flops": float((2 * n ** 3 / 3 if case["form"] != "bj" else 60 * n * n) + 10 * n * n)}
    if kind == "ell_batch":
        pairs = sum(k * k for k in _sizes(case, 0))
        return {"bytes": 8.0 * sum(34 * k for k in _sizes(case, 0)), "flops": 30000.0 * pairs + 60 * 576 * pairs}
    if kind == "cube":
        el, pts = 6 * case["n_face"] ** 2, case["grid"] ** 3
        nn = el + 2
        n = 3 * nn + case["layout"] * case["num"]
        return {"bytes": 8.0 * (3 * nn + 28 * el + 4 * case["num"] + n + 9 * pts),
                "flops": 2 * n ** 3 / 3 + 64.0 * el * (115 * pts + 300 * nn + 100 * case["layout"] * case["num"])}
    e = 16 * case["num"]
    macs = case["num"] * (640 + 3 * 128 * 64) + e * (4 * 135 * 64 + 128)
    return {"bytes": 4.0 * (case["num"] * (10 + 24 * case["nrhs"]) + e * (8 + 48 * case["nrhs"]) + 7 * 60418), "flops": 6.0 * macs}


# --------------------------------------------------------------------------- exact values (spheres, training step)
_IJ = [(i, j) for i in range(3) for j in range(i, 3)]
_V = 4 * math.pi / 3


def _units(layout):
    """(order, i, j, moments, multiplier) of every unknown of a sphere."""
    u = [(0, i, j, (), 1) for i, j in _IJ] + [(1, i, j, (p,), 1) for i, j in _IJ for p in range(3)]
    if layout > 24:
        u += [(2, i, j, (p, q), 2 if layout == 60 and p != q else 1) for i, j in _IJ for p in range(3)
              for q in range(p if layout == 60 else 0, 3)]
    return u


def _alpha(idx):
    return (idx.count(0), idx.count(1), idx.count(2))


def _outside(name, mom):
    """Potential phi (density / r) or psi (density * r) of the unit sphere: {(power of r, derivative indices): factor}."""
    phi = name == "phi"
    if len(mom) == 0:
        return {(-1, ()): _V} if phi else {(1, ()): _V, (-1, ()): _V / 5}
    if len(mom) == 1:
        return {(-1, mom): -_V / 5} if phi else {(1, mom): -_V / 5, (-1, mom): -_V / 35}
    out = {(-1, mom): _V / 35} if phi else {(1, mom): _V / 35, (-1, mom): _V / 315}
    if mom[0] == mom[1]:
        out.update({(-1, ()): _V / 5} if phi else {(1, ()): _V / 5, (-1, ()): _V / 35})
    return out


def _poly_mul(p, q):
    out = {}
    for (a, x), (b, y) in itertools.product(p.items(), q.items()):
        k = tuple(s + t for s, t in zip(a, b))
        out[k] = out.get(k, 0.0) + x * y
    return out


def _poly_add(*terms):
    out = {}
    for f, p in terms:
        for k, v in p.items():
            out[k] = out.get(k, 0.0) + f * v
    return out


def _poly_d(p, idx):
    for i in idx:
        q = {}
        for k, v in p.items():
            if k[i]:
                q[k[:i] + (k[i] - 1,) + k[i + 1:]] = v * k[i]
        p = q
    return p


_ONE = {(0, 0, 0): 1.0}
_R2 = {(2, 0, 0): 1.0, (0, 2, 0): 1.0, (0, 0, 2): 1.0}


@functools.lru_cache(None)
def _inside(name, mom):
    """The same potentials inside the unit sphere, up to terms that the strains do not see, as polynomials."""
    pi, r4 = math.pi, _poly_mul(_R2, _R2)
    x = _ONE
    for p in mom:
        x = _poly_mul(x, {tuple(int(k == p) for k in range(3)): 1.0})
    d = 1.0 if len(mom) == 2 and mom[0] == mom[1] else 0.0
    if len(mom) == 0:
        return {k: -2 * pi / 3 * v for k, v in _R2.items()} if name == "phi" else _poly_add((2 * pi / 3, _R2), (-pi / 15, r4))
    if len(mom) == 1:
        rad = _poly_add((2 * pi / 3, _ONE), (-2 * pi / 5, _R2)) if name == "phi" else _poly_add((2 * pi / 15, _R2), (-pi / 35, r4))
        return _poly_mul(x, rad)
    a, b, c = -2 * pi / 7, pi / 35, 2 * pi / 5
    if name == "phi":
        return _poly_add((1, _poly_mul(x, _poly_add((a, _R2), (c, _ONE)))), (d * b, r4), (-d * c / 3, _R2))
    c1, c3 = a / 18, c / 7
    return _poly_add((1, _poly_mul(x, _poly_add((c1, r4), (c3, _R2)))), (d * (b - c1) / 21, _poly_mul(_R2, r4)),
                     (d * (-2 * c / 3 - 2 * c3) / 20, r4))


def _strain_terms(i, j, k, l):
    """D_ijkl as a sum over derivatives of psi and phi: (factor, potential, derivative indices)."""
    t = [(1.0, "psi", (k, l, i, j))]
    if k == l:
        t.append((-2 * NU0, "phi", (i, j)))
    for hit, rest in ((i == l, (k, j)), (j == l, (k, i)), (i == k, (l, j)), (j == k, (l, i))):
        if hit:
            t.append((-(1 - NU0), "phi", rest))
    return [(f / (8 * math.pi * (1 - NU0)), n, d) for f, n, d in t]


@functools.lru_cache(None)
def _alphas(order):
    return [(a, b, n - a - b) for n in range(order + 1) for a in range(n, -1, -1) for b in range(n - a, -1, -1)]


def _d_outside(i, j, unit, der):
    """{(power, derivative): factor} of strain (i, j) and its derivative `der` for one eigenstrain unknown."""
    _, k, l, mom, _ = unit
    out = {}
    for f, name, d in _strain_terms(i, j, k, l):
        for (s, m), v in _outside(name, mom).items():
            key = (s, _alpha(d + m + der))
            out[key] = out.get(key, 0.0) + f * v
    return out


def _d_inside(i, j, unit, der):
    _, k, l, mom, _ = unit
    return _poly_add(*[(f, _poly_d(_inside(name, mom), d + der)) for f, name, d in _strain_terms(i, j, k, l)])


def _row(dlam, dmu, i, j, get):
    """sum_kl (C0 - C1)_ijkl D_kl for a getter of D."""
    t = [(2 * dmu, get(i, j))]
    if i == j:
        t += [(dlam, get(k, k)) for k in range(3)]
    return _poly_add(*t)


def _lame(E, nu):
    mu = E / (2 * (1 + nu))
    return 2 * mu * nu / (1 - 2 * nu), mu


def _scaled_blocks(E1, layout):
    """The pair block of unit spheres divided by mu0, as a matrix over [derivatives of r | of 1/r], and the self block."""
    (l0, m0), (l1, m1) = _lame(E0, NU0), _lame(E1, NU1)
    units, al = _units(layout), _alphas(4 + (2 if layout == 24 else 4))
    col = {(s, a): (0 if s == 1 else len(al)) + n for s in (1, -1) for n, a in enumerate(al)}
    out = np.zeros((layout * layout, 2 * len(al)))
    own = np.zeros((layout, layout))
    for r, (ro, i, j, der, _) in enumerate(units):
        for c, unit in enumerate(units):
            co, m, n, mom, mult = unit
            fac = (0.5 if ro == 2 else 1.0) * (1 if m == n else 2)
            for key, v in _row((l0 - l1) / m0, (m0 - m1) / m0, i, j, lambda a, b: _d_outside(a, b, unit, der)).items():
                out[r * layout + c, col[key]] -= fac * mult * v
            v = _row((l0 - l1) / m0, (m0 - m1) / m0, i, j, lambda a, b: _d_inside(a, b, unit, der)).get((0, 0, 0), 0.0)
            own[r, c] = -fac * mult * v
            if ro == co and der == mom:
                own[r, c] += (l0 / m0 * (i == j) * (m == n) + (i == m) * (j == n)
                              + (i == n) * (j == m)) * (1 if m == n else 2)
    return torch.from_numpy(out).cuda(), torch.from_numpy(own).cuda()


def _derivatives(x, order):
    """All derivatives up to `order` of r, then of 1/r, at the rows of x: (2 * count, n)."""
    al = _alphas(order)
    pos = {a: k for k, a in enumerate(al)}
    n = x.shape[0]
    xs = [x[:, 0].contiguous(), x[:, 1].contiguous(), x[:, 2].contiguous()]
    inv = (xs[0] ** 2 + xs[1] ** 2 + xs[2] ** 2).rsqrt()
    low = {}                                         # derivatives of r^(s-2) while those of r^s are made
    for s in range(-1 - 2 * order, 2, 2):
        top = order + min(0, (s + 1) // 2)
        cur = {(0, 0, 0): inv ** (-s)}
        for a in _alphas(top)[1:]:
            i = next(t for t in range(3) if a[t])
            b = a[:i] + (a[i] - 1,) + a[i + 1:]
            v = xs[i] * low[b]
            if b[i]:
                v = v + b[i] * low[b[:i] + (b[i] - 1,) + b[i + 1:]]
            cur[a] = s * v
        low = cur
        if s == -1:
            minus = cur
    out = torch.empty((2 * len(al), n), dtype=torch.float64, device=x.device)
    for a, k in pos.items():
        out[k], out[len(al) + k] = cur[a], minus[a]
    return out


def _matrix(c, layout):
    """Scaled system Dr A Dc of one realisation (unknowns times radius^order, rows over mu0), row-major."""
    blk, own = _scaled_blocks(c.E1, layout)
    cen, rad = torch.from_numpy(c.centers).cuda(), torch.from_numpy(c.radius).cuda()
    n = c.num
    order = torch.tensor([u[0] for u in _units(layout)], dtype=torch.float64, device="cuda")
    A = torch.empty((n, layout, n, layout), dtype=torch.float64, device="cuda")
    step = max(1, 400_000 // n)
    for h in range(0, n, step):
        k = min(step, n - h)
        x = (cen[:, None] - cen[None, h:h + k]) / rad[None, h:h + k, None]
        same = torch.arange(n, device="cuda")[:, None] == torch.arange(h, h + k, device="cuda")[None]
        x = torch.where(same[..., None], torch.full_like(x, 9.0), x)
        b = (blk @ _derivatives(x.reshape(-1, 3), 6 if layout == 24 else 8)).reshape(layout, layout, n, k)
        b = b * ((rad[:, None] / rad[None, h:h + k])[None] ** order[:, None, None])[:, None]
        A[:, :, h:h + k, :] = b.permute(2, 0, 3, 1)
        at = torch.arange(h, h + k, device="cuda")
        A[at, :, at, :] = own
    return A.reshape(n * layout, n * layout)


def _solve(c, layout):
    """Eigenstrain coefficients of one realisation under SIG: a direct solve, or GMRES(300) where that takes too long."""
    A = _matrix(c, layout)
    (l0, m0), (l1, m1) = _lame(c.E0, c.nu0), _lame(c.E1, c.nu1)
    s = np.array([[SIG[0], SIG[1], SIG[2]], [SIG[1], SIG[3], SIG[4]], [SIG[2], SIG[4], SIG[5]]])
    eps = ((1 + c.nu0) * s - c.nu0 * np.trace(s) * np.eye(3)) / c.E0
    r = ((l0 - l1) * np.trace(eps) * np.eye(3) + 2 * (m0 - m1) * eps) / m0
    b = torch.zeros((c.num, layout), dtype=torch.float64, device="cuda")
    b[:, :6] = torch.tensor([r[i, j] for i, j in _IJ], dtype=torch.float64, device="cuda")
    b = b.reshape(-1)
    if len(b) <= 20000:
        y = torch.linalg.solve(A, b)
        y = y + torch.linalg.solve(A, b - A @ y) if len(b) <= 6000 else y
    else:
        inv = torch.linalg.inv(A[:layout, :layout])
        prec = lambda v: (v.reshape(-1, layout) @ inv.T).reshape(-1)
        y, beta = torch.zeros_like(b), b.norm()
        for _ in range(4):
            res = b - A @ y
            if res.norm() < 3e-15 * beta:
                break
            q, hess = [res / res.norm()], []
            for k in range(40):
                w = A @ prec(q[-1])
                Q = torch.stack(q)
                h = Q @ w
                w = w - h @ Q
                h2 = Q @ w
                w = w - h2 @ Q
                hess.append(torch.cat([h + h2, w.norm()[None]]).cpu().numpy())
                q.append(w / w.norm())
                if hess[-1][-1] < 1e-15:
                    break
            H = np.zeros((len(hess) + 1, len(hess)))
            for k, h in enumerate(hess):
                H[:len(h), k] = h
            rhs = np.zeros(len(hess) + 1)
            rhs[0] = float(res.norm())
            z = np.linalg.lstsq(H, rhs, rcond=None)[0]
            y = y + prec(torch.from_numpy(z).cuda() @ torch.stack(q[:-1]))
    a = torch.from_numpy(c.radius).cuda()[:, None]
    order = torch.tensor([u[0] for u in _units(layout)], dtype=torch.float64, device="cuda")
    return (y.reshape(c.num, layout) / a ** order).reshape(-1)


def _moduli(cs, x, layout):
    """Effective modulus and mean strain of each realisation."""
    strain, at = [], 0
    s = np.array([[SIG[0], SIG[1], SIG[2]], [SIG[1], SIG[3], SIG[4]], [SIG[2], SIG[4], SIG[5]]])
    for c in cs:
        e = x[at:at + c.num * layout].reshape(c.num, layout).cpu().numpy()
        at += c.num * layout
        mean = e[:, :6].copy()
        for k, (o, i, j, mom, _) in enumerate(_units(layout)):
            if o == 2 and mom[0] == mom[1]:
                mean[:, _IJ.index((i, j))] += c.radius ** 2 / 5 * e[:, k]
        eps = ((1 + c.nu0) * s - c.nu0 * np.trace(s) * np.eye(3)) / c.E0
        strain.append(np.array([eps[i, j] for i, j in _IJ]) + (_V * c.radius ** 3) @ mean / _side(c) ** 3)
    strain = np.array(strain)
    return SIG[5] / strain[:, 5], strain


def _stress(c, layout, e, pts):
    """Stresses at pts (n x 3) from the coefficients e (num x layout) under SIG."""
    units, order = _units(layout), 4 + (1 if layout == 24 else 2)
    al = _alphas(order)
    col = {(s, a): (0 if s == 1 else len(al)) + n for s in (1, -1) for n, a in enumerate(al)}
    mono = [(a, b, n - a - b) for n in range(3) for a in range(n, -1, -1) for b in range(n - a, -1, -1)]
    out = np.zeros((6, layout, len(col)))
    ins = np.zeros((6, layout, len(mono)))
    for r, (i, j) in enumerate(_IJ):
        for k, unit in enumerate(units):
            f = (1 if unit[1] == unit[2] else 2) * unit[4]
            for key, v in _d_outside(i, j, unit, ()).items():
                out[r, k, col[key]] += f * v
            for key, v in _d_inside(i, j, unit, ()).items():
                if sum(key) <= 2:
                    ins[r, k, mono.index(key)] += f * v
            if (unit[1], unit[2]) == (i, j):   # the local eigenstrain comes off inside
                o, mom = unit[0], unit[3]
                if not (layout == 78 and o == 2 and mom[0] > mom[1]):
                    ins[r, k, mono.index(_alpha(mom))] -= 2 if o == 2 and mom[0] != mom[1] else 1
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    a = c.radius
    es = dev(np.asarray(e).reshape(c.num, layout) * a[:, None] ** np.array([u[0] for u in units])[None])
    w_out = torch.einsum("hk,rkc->hrc", es, dev(out))
    w_in = torch.einsum("hk,rkc->hrc", es, dev(ins))
    cen, pts = dev(c.centers), dev(pts)
    strain = torch.zeros((6, pts.shape[0]), dtype=torch.float64, device="cuda")
    for h in range(c.num):
        x = (pts - cen[h]) / a[h]
        inside = (x * x).sum(1) <= 1
        d = _derivatives(torch.where(inside[:, None], torch.full_like(x, 9.0), x), order)
        v = w_out[h] @ d
        if bool(inside.any()):
            y = x[inside]
            m = torch.stack([y[:, 0] ** p * y[:, 1] ** q * y[:, 2] ** s for p, q, s in mono])
            v[:, inside] = w_in[h] @ m
        strain += v
    l0, m0 = _lame(c.E0, c.nu0)
    tr = strain[0] + strain[3] + strain[5]
    s = 2 * m0 * strain + dev(np.array(SIG))[:, None]
    for r in (0, 3, 5):
        s[r] += l0 * tr
    return s.T.contiguous()


def exact(case, seed):
    """FP64 values of run()'s outputs by torch alone.  None where it would take too long (20,000 spheres, long stress
    grids), for the boundary elements of the cube and for ellipsoids, whose blocks have no closed form this short."""
    kind = case["kind"]
    if kind == "solve":
        if case["num"] > 2000:
            return None
        cs, layout = [_sphere_case(case["num"], case["vf"], case["contrast"], seed)], 24
    elif kind == "batch":
        cs, layout = _realisations(case, seed), case["layout"]
    elif kind == "dense":
        cs, layout = [_sphere_case(case["num"], case["vf"], 5.714, seed)], case["layout"]
    elif kind == "host":
        c = _sphere_case(case["num"], case["vf"], case["contrast"], seed, grid=case["grid"])
        x = _solve(c, 24)
        if case["num"] * case["grid"] ** 3 > 6e8:
            return dict(x=x, stress=None)
        return dict(x=x.cpu().numpy(), stress=_stress(c, 24, x.cpu().numpy(), c.points).cpu().numpy())
    elif kind == "field":
        c, e = _field_inputs(case, seed)
        side = _side(c)
        ax = [(np.arange(case[n]) + 0.5) * side / case[n] for n in ("nx", "ny", "nz")]
        z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        return dict(stress=_stress(c, case["layout"], e, np.stack([x.ravel(), y.ravel(), z.ravel()], 1)))
    elif kind == "train":
        return _exact_train(case, seed)
    else:
        return None
    x = torch.cat([_solve(c, layout) for c in cs])
    e, strain = _moduli(cs, x, layout)
    return dict(x=x, e_eff=e, strain=strain)


def _exact_train(case, seed):
    s = {k: (v.double() if v.is_floating_point() else v.long()).cuda() for k, v in _graph(case, seed).items()}
    num, h = case["num"], 64
    p = s["params"].clone().requires_grad_(True)
    at, layers = 0, []
    for fan_in, fan_out in [(10, h)] + [(2 * h + 7, h), (2 * h, h)] * 3 + [(2 * h + 7, h), (h, 2)]:
        layers.append((p[at:at + fan_in * fan_out].reshape(fan_in, fan_out), p[at + fan_in * fan_out:at + (fan_in + 1) * fan_out]))
        at += (fan_in + 1) * fan_out
    lin = lambda k, v: v @ layers[k][0] + layers[k][1]
    edge = lambda v: torch.cat([v[:, None].expand(num, 16, h), v[s["nbr"]], s["ef"]], 2)
    v = torch.relu(lin(0, s["xn"]))
    for k in range(3):
        m = torch.relu(lin(1 + 2 * k, edge(v))).mean(1)
        v = v + torch.relu(lin(2 + 2 * k, torch.cat([v, m], 1)))
    w = lin(8, torch.relu(lin(7, edge(v))))
    u = s["u"].reshape(case["nrhs"], num, 16, 2, 24)
    loss = ((s["z"] + (w[None, ..., None] * u).sum((2, 3))) ** 2).sum()
    loss.backward()
    b1, b2, step, lr = 0.9, 0.999, 20, 2e-3
    m = b1 * s["m"] + (1 - b1) * p.grad
    q = b2 * s["v"] + (1 - b2) * p.grad ** 2
    new = s["params"] * (1 - lr * 1e-4) - lr * (m / (1 - b1 ** step)) / ((q / (1 - b2 ** step)).sqrt() + 1e-8)
    return dict(loss=float(loss.detach()), grad=p.grad, params=new, m=m, v=q)
