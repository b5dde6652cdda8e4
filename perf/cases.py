"""The workloads this library is timed on, through its public entry points.

A user of the library assembles the residual and the Jacobian of a mesh at a
state, many times over: in FP64 or mixed precision, into device or host
memory, one mesh at a time or many in one batched launch; or lets the library
run a whole Newton load step; or trains and evaluates the small network that
predicts the initial guess of a load step.  Each case is one such call.  All
inputs are synthetic and seeded: box meshes with perturbed interior nodes and
a smooth deformation of them.

``exact`` restates the same element integrals in plain FP64 torch tensor
algebra (the textbook index notation, assembled by sorting the (row, column)
pairs of all elements).
"""
import math

import numpy as np
import torch

from cm_gb300 import EquationsSetBatch, FiniteElasticityEquationsSet, create_equations_sets
from cm_gb300.mesh import GUCCIONE, MR, Mesh
from cm_gb300.warmstart import MLP

DEV = "cuda"
WIDTHS = (4, 256, 256, 256, 64)  # the warm-start network: four load/material parameters to 64 POD modes


def _box(name, kind, ex, ey, ez, nxi=3, pressure="node", law="mr", load=False):
    return {"name": name, "kind": kind, "ex": ex, "ey": ey, "ez": ez, "nxi": nxi, "pressure": pressure,
            "law": law, "load": load}


def listed():
    return [
        # The plain method's smallest problem: the FP64 Jacobian and residual of a 4x4x4 trilinear cube.
        _box("fp64_trilinear_4x4x4", "fp64", 4, 4, 4, nxi=2, pressure="element"),
        # The FP64 Jacobian of a Newton step of the plain method, at the warm-start study's mesh size.
        _box("fp64_triquadratic_16", "fp64", 16, 16, 16),
        # A residual inside a line search on a small, odd-sized mesh: launch latency counts.
        _box("residual_9x7x8", "residual", 9, 7, 8),
        # The residual of the large mesh.
        _box("residual_32", "residual", 32, 32, 32),
        # Mixed-precision assembly on a mesh too small to fill the GPU (the load-step bench's size).
        _box("mixed_9x7x8", "mixed", 9, 7, 8),
        # The headline assembly: 32^3 triquadratic displacement, trilinear nodal pressure, Mooney-Rivlin.
        _box("mixed_32", "mixed", 32, 32, 32),
        # The cardiac-style slab: Guccione law, a fibre field, cavity pressure on the z = 0 face; ragged sizes.
        _box("mixed_slab_33x31x9", "mixed", 33, 31, 9, law="guccione", load=True),
        # The end-to-end call of a host code: page-locked host state in, assembled system out.
        _box("mixed_host_16", "mixed_host", 16, 16, 16),
        # Many meshes of uneven size, element type and material in one batched assembly, replayed from a graph.
        {"name": "batch_24_boxes", "kind": "batch", "members": 24, "lo": 4, "hi": 24},
        # One whole load increment by the library's Newton solver.
        _box("newton_6x5x4", "newton", 6, 5, 4),
        # One training step of the warm-start network (forward, backward, Adam) on a minibatch.
        {"name": "train_256", "kind": "train", "rows": 256},
        # The network's prediction for a set of held-out problems.
        {"name": "infer_256", "kind": "infer", "rows": 256},
    ]


def _edges(rng, lo, hi):
    """Three edge counts whose product is log-uniform in [lo, hi], with aspect ratios up to about 3."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
    s = n ** (1.0 / 3.0)
    return [max(2, round(s * f)) for f in (a, b, 1.0 / (a * b))]


def draw(rng):
    kind = rng.choice(["fp64", "residual", "residual", "mixed", "mixed", "mixed", "mixed_host", "batch", "newton",
                       "train", "infer"])
    if kind == "train":
        return {"kind": kind, "rows": rng.randint(32, 512)}
    if kind == "infer":
        return {"kind": kind, "rows": round(math.exp(rng.uniform(0.0, math.log(2048))))}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(4, 28), "lo": 4, "hi": rng.randint(10, 24)}
    nxi = rng.choice([2, 3, 3])
    if kind == "newton":
        e = _edges(rng, 60, 130) if nxi == 3 else _edges(rng, 64, 400)
    else:
        e = _edges(rng, 64, 4096 if kind == "fp64" else (8000 if kind == "mixed_host" else 24000))
    law = "mr" if kind == "newton" else rng.choice(["mr", "mr", "guccione"])
    pressure = "node" if nxi == 3 else "element" if kind == "newton" else rng.choice(["element", "node"])
    c = _box("", kind, *e, nxi=nxi, pressure=pressure, law=law, load=law == "guccione" and rng.random() < 0.5)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

def _mesh_arrays(ex, ey, ez, lengths, nxi, pressure, perturb, rng):
    """Connectivity (elements and nodes x fastest), node coordinates and grid of a box."""
    dims = np.array([ex, ey, ez])
    grid = (nxi - 1) * dims + 1
    e = np.arange(ex * ey * ez)
    e0 = np.stack([e % ex, (e // ex) % ey, e // (ex * ey)], 1) * (nxi - 1)
    a = np.arange(nxi ** 3)
    loc = np.stack([a % nxi, (a // nxi) % nxi, a // nxi ** 2], 1)
    ijk = e0[:, None, :] + loc[None, :, :]
    elem_u = (ijk[..., 0] + grid[0] * (ijk[..., 1] + grid[1] * ijk[..., 2])).astype(np.int32)
    nu = int(grid.prod())
    n = np.arange(nu)
    g = np.stack([n % grid[0], (n // grid[0]) % grid[1], n // (grid[0] * grid[1])])
    X = g * (np.asarray(lengths) / (grid - 1))[:, None]
    if perturb:
        inner = ((g > 0) & (g < (grid - 1)[:, None])).all(0)
        h = np.asarray(lengths) / dims
        X[:, inner] += rng.uniform(-perturb, perturb, size=(3, int(inner.sum()))) * h[:, None]
    elem_p = None
    if pressure == "node":
        corner = np.nonzero((loc % (nxi - 1) == 0).all(1))[0]
        users = elem_u[:, corner]
        elem_p = np.searchsorted(np.unique(users), users).astype(np.int32)
    return elem_u, elem_p, X, g, tuple(int(v) for v in grid)


def _one(ex, ey, ez, nxi, pressure, law, load, rng, perturb=0.1, lengths=(1.0, 1.0, 1.0), stretch=(1.0, 1.3),
         shear=(0.0, 0.2)):
    """A mesh, its materials and a deformed state, as plain arrays."""
    if law == "guccione":  # millimetres and kilopascals; a stiff exponential law sees small strains
        lengths, stretch, shear = (0.625 * ex, 0.625 * ey, 0.625 * ez), (1.0, 1.05), (0.0, 0.02)
    elem_u, elem_p, X, g, grid = _mesh_arrays(ex, ey, ez, lengths, nxi, pressure, perturb, rng)
    nu = X.shape[1]
    m = {"dims": (ex, ey, ez), "lengths": tuple(lengths), "nxi": nxi, "pressure": pressure, "law": law, "grid": grid,
         "elem_u": elem_u, "elem_p": elem_p, "X": X, "g": g, "fibre": None, "surf": None}
    if law == "guccione":
        m["materials"] = np.array([math.exp(rng.uniform(math.log(0.5), math.log(2.0))), 18.5, 3.58, 1.63])
        ang = np.deg2rad(-60.0 + 120.0 * X[2] / lengths[2] + rng.uniform(-5.0, 5.0, size=nu))
        m["fibre"] = np.stack([ang, np.zeros(nu), np.zeros(nu)])
    else:
        m["materials"] = np.exp(rng.uniform(math.log(0.5), math.log(10.0), size=2))
    if load:
        m["surf"] = np.zeros((3, nu))
        m["surf"][2, g[2] == 0] = rng.uniform(0.25, 2.0)
    lam, gam = rng.uniform(*stretch), rng.uniform(*shear)
    z = X / math.sqrt(lam)
    z[0] = lam * X[0] + gam * X[1]
    h = min(l / d for l, d in zip(lengths, (ex, ey, ez))) / (nxi - 1)
    z = z + rng.uniform(-0.02, 0.02, size=z.shape) * h
    n_p = len(elem_u) if elem_p is None else int(elem_p.max()) + 1
    p = rng.uniform(-2.0, -1.0) * (1.0 + 0.1 * rng.uniform(-1.0, 1.0, size=n_p))
    m["x"] = np.concatenate([z.ravel(), p])
    return m


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 17])
    if case["kind"] == "batch":
        shapes = np.random.default_rng(case["members"])  # the sizes belong to the case, the values to the seed
        out = []
        for _ in range(case["members"]):
            e = [int(v) for v in shapes.integers(case["lo"], case["hi"] + 1, size=3)]
            quad = bool(shapes.integers(0, 2))
            out.append(_one(*e, 3 if quad else 2, "node" if quad else "element", "mr", False, rng, perturb=0.0,
                            lengths=tuple(rng.uniform(0.5, 2.0, size=3)), shear=(0.0, 0.0)))
        return out
    m = _one(case["ex"], case["ey"], case["ez"], case["nxi"], case["pressure"], case["law"], case["load"], rng)
    if case["kind"] == "newton":
        # a first load increment: the x = 0 face clamped, the x = 1 face moved a little from the undeformed state
        nu, X, g = m["X"].shape[1], m["X"], m["g"]
        lam, gam = rng.uniform(1.01, 1.03), rng.uniform(0.0, 0.02)
        left, right = np.nonzero(g[0] == 0)[0], np.nonzero(g[0] == m["grid"][0] - 1)[0]
        m["dofs"] = np.concatenate([c * nu + left for c in range(3)] + [c * nu + right for c in range(3)])
        m["values"] = np.concatenate([X[0, left], X[1, left], X[2, left], lam * X[0, right],
                                      X[1, right] + gam * X[0, right], X[2, right]])
        m["x"] = np.concatenate([X.ravel(), np.zeros(len(m["x"]) - 3 * nu)])
    return m


def _mesh(m):
    return Mesh(dims=m["dims"], lengths=m["lengths"], nxi_u=m["nxi"], p_mode=1 if m["pressure"] == "node" else 0,
                law=MR if m["law"] == "mr" else GUCCIONE, elem_u=m["elem_u"], elem_p=m["elem_p"], X=m["X"],
                materials=m["materials"], fibre=m["fibre"], grid_u=m["grid"])


def _training(case, seed):
    """Network weights in the middle of a training run (Adam moments of the gradients' size), and a minibatch."""
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    n = sum(i * o + o for i, o in zip(WIDTHS[:-1], WIDTHS[1:]))
    x = rnd(case["rows"], WIDTHS[0])
    basis = rnd(WIDTHS[0], WIDTHS[-1])
    y = torch.tanh(x @ basis) + 0.1 * rnd(case["rows"], WIDTHS[-1])
    return {"bias": 0.1 * rnd(n), "m": 1e-4 * rnd(n), "v": 1e-7 * (0.5 + torch.rand(n, generator=g)), "x": x, "y": y,
            "weights": [rnd(o, i) * math.sqrt(2.0 / (i + o)) for i, o in zip(WIDTHS[:-1], WIDTHS[1:])]}


LR, STEP = 1e-3, 200


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "infer"):
        t = _training(case, seed)
        net = MLP(WIDTHS, seed=seed, device=DEV)
        net.flat.copy_(t["bias"])
        for l, w in enumerate(t["weights"]):
            net.W(l).copy_(w)
        net.m.copy_(t["m"])
        net.v.copy_(t["v"])
        net.step = STEP
        return {"kind": kind, "net": net, "x": t["x"].to(DEV), "y": t["y"].to(DEV)}
    if kind == "batch":
        ms = _inputs(case, seed)
        sets = create_equations_sets([_mesh(m) for m in ms])
        batch = EquationsSetBatch(sets)
        xs = [torch.from_numpy(m["x"]).to(DEV) for m in ms]
        flat, views = [], []
        for sizes, dt in (([s.nnz_uu for s in sets], torch.float32), ([s.nnz_coupling for s in sets], torch.float64),
                          ([s.ndofs for s in sets], torch.float64)):
            at, total = _places(sizes)
            flat.append(torch.zeros(total, dtype=dt, device=DEV))
            views.append([flat[-1][a:a + n] for a, n in zip(at, sizes)])
        batch.autotune(xs, *views, repeats=3)
        batch.capture(xs, *views)
        return {"kind": kind, "sets": sets, "batch": batch, "xs": xs, "views": views, "out": flat}
    m = _inputs(case, seed)
    es = FiniteElasticityEquationsSet(_mesh(m))
    if m["surf"] is not None:
        es.set_surface_pressure(m["surf"])
    s = {"kind": kind, "es": es}
    if kind == "mixed_host":
        pinned = lambda n, dt: torch.zeros(n, dtype=dt).pin_memory().numpy()  # noqa: E731
        s["x"] = pinned(es.ndofs, torch.float64)
        s["x"][:] = m["x"]
        s["out"] = (pinned(es.nnz_uu, torch.float32), pinned(es.nnz_coupling, torch.float64),
                    pinned(es.ndofs, torch.float64))
        return s
    s["x"] = torch.from_numpy(m["x"]).to(DEV)
    new = lambda n, dt=torch.float64: torch.empty(n, dtype=dt, device=DEV)  # noqa: E731
    if kind == "newton":
        s["dofs"], s["values"] = m["dofs"].astype(np.int32), m["values"]
    elif kind == "mixed":
        s["out"] = (new(es.nnz_uu, torch.float32), new(es.nnz_coupling), new(es.ndofs))
    elif kind == "fp64":
        s["out"] = (new(es.nnz), new(es.ndofs))
    else:
        s["out"] = new(es.ndofs)
    return s


def _places(sizes):
    """Where each member's array begins in one flat buffer (multiples of 64 entries), and the total."""
    at, n = [], 0
    for k in sizes:
        at.append(n)
        n += -(-k // 64) * 64
    return at, n


def run(state):
    kind = state["kind"]
    if kind == "train":
        net = state["net"]
        loss = net.loss_and_grad(state["x"], state["y"])
        net.adam_step(LR)
        return {"loss": loss, "grad": net.grad, "weights": net.flat}
    if kind == "infer":
        return state["net"].infer_bf16(state["x"])
    if kind == "batch":
        state["batch"].replay(state["xs"][0])
        return state["out"]
    es = state["es"]
    if kind == "newton":
        x = state["x"].clone()
        es.newton_load_step(x, state["dofs"], state["values"])
        return x
    if kind == "residual":
        return es.residual_evaluate(state["x"], state["out"])
    if kind == "fp64":
        values, r = state["out"]
        es.jacobian_evaluate(state["x"], values, r)
    else:
        es.jacobian_evaluate_mixed(state["x"], *state["out"])
    return state["out"]


# -------------------------------------------------------------------- work

def _pattern_size(grid, dims, nxi, pressure):
    """(displacement nodes, pressure unknowns, displacement-block entries, coupling entries) of a box."""
    def pairs(na, nb):  # (a, b) index pairs sharing an element along one edge, a on na- and b on nb-point lines
        return lambda e: sum(len({b for k in range(e) if (na - 1) * k <= a <= (na - 1) * (k + 1)
                                  for b in range((nb - 1) * k, (nb - 1) * (k + 1) + 1)})
                             for a in range((na - 1) * e + 1))
    prod = lambda f: math.prod(f(e) for e in dims)  # noqa: E731
    nu = math.prod(grid)
    uu = 9 * prod(pairs(nxi, nxi))
    if pressure == "node":
        n_p = math.prod(e + 1 for e in dims)
        return nu, n_p, uu, 2 * 3 * prod(pairs(nxi, 2)) + prod(pairs(2, 2))
    ne = math.prod(dims)
    return nu, ne, uu, 2 * 3 * ne * nxi ** 3 + ne


def _element_flops(nxi, pressure, jacobian):
    """Sum-factorised element integrals (multiply and add counted apart)."""
    n, G = nxi, 3
    stages = n * n * G + n * G * G + G ** 3
    grad = 3 * 3 * stages * n
    gauss = 27 * (300 + (900 if jacobian else 0))
    res = 9 * (G * G * n + G * n * n + n ** 3) * G
    uu = 6 * (9 * n * n * G ** 3 + 9 * n ** 4 * G * G + 4 * n ** 6 * G) if jacobian else 0
    cp = (8 if pressure == "node" else 1) * 3 * n ** 3 * 6 if jacobian else 0
    return 2 * (grad + res + uu + cp) + gauss


def _box_work(kind, dims, nxi, pressure, fibre):
    grid = [(nxi - 1) * e + 1 for e in dims]
    ne = math.prod(dims)
    nu, n_p, uu, cp = _pattern_size(grid, dims, nxi, pressure)
    nd = 3 * nu + n_p
    bytes_in = 8 * nd + 8 * 3 * nu * (2 if fibre else 1) + 4 * ne * (nxi ** 3 + (8 if pressure == "node" else 0))
    out = 8 * nd
    if kind == "fp64":
        out += 8 * (uu + cp)
    elif kind in ("mixed", "mixed_host", "batch"):
        out += 4 * uu + 8 * cp
    flops = ne * _element_flops(nxi, pressure, kind != "residual")
    if kind == "newton":  # three Newton steps: a Jacobian written and read by thirty matrix-vector products in each
        out += 3 * 8 * (uu + cp) * 31
        flops = 3 * flops + 3 * 30 * 2 * (uu + cp)
    return bytes_in + out, flops


def work(case):
    kind = case["kind"]
    params = sum(i * o + o for i, o in zip(WIDTHS[:-1], WIDTHS[1:]))
    macs = sum(i * o for i, o in zip(WIDTHS[:-1], WIDTHS[1:]))
    if kind == "train":  # weights and both moments read and written, the gradient written
        return {"bytes": 28 * params + 4 * case["rows"] * (WIDTHS[0] + WIDTHS[-1]), "flops": 6 * macs * case["rows"]}
    if kind == "infer":
        return {"bytes": 2 * params + 4 * case["rows"] * (WIDTHS[0] + WIDTHS[-1]), "flops": 2 * macs * case["rows"]}
    if kind == "batch":
        b = f = 0
        shapes = np.random.default_rng(case["members"])
        for _ in range(case["members"]):
            e = [int(v) for v in shapes.integers(case["lo"], case["hi"] + 1, size=3)]
            quad = bool(shapes.integers(0, 2))
            one = _box_work(kind, e, 3 if quad else 2, "node" if quad else "element", False)
            b, f = b + one[0], f + one[1]
        return {"bytes": b, "flops": f}
    b, f = _box_work(kind, (case["ex"], case["ey"], case["ez"]), case["nxi"], case["pressure"],
                     case["law"] == "guccione")
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact

def _lagrange(n, t):
    """Values and derivatives of the 1-D Lagrange basis with n equally spaced nodes on [0, 1] at the points t."""
    node = torch.linspace(0, 1, n, dtype=torch.float64, device=t.device)
    c = torch.linalg.inv(node[:, None] ** torch.arange(n, device=t.device))  # monomial coefficients, [power][basis]
    k = torch.arange(n, device=t.device)
    val = (t[:, None] ** k) @ c
    der = (k * t[:, None] ** (k - 1).clamp(min=0)) @ c
    return val, der


def _basis(n):
    """N [27, n^3], dN/dxi [27, n^3, 3] at the 3x3x3 Gauss points (x fastest) and the weights."""
    t = torch.tensor([0.5 - math.sqrt(0.15), 0.5, 0.5 + math.sqrt(0.15)], dtype=torch.float64, device=DEV)
    w = torch.tensor([5.0, 8.0, 5.0], dtype=torch.float64, device=DEV) / 18.0
    v, d = _lagrange(n, t)
    tensor = lambda a, b, c: torch.einsum("ga,hb,ic->ihgcba", a, b, c).reshape(27, n ** 3)  # noqa: E731
    return (tensor(v, v, v), torch.stack([tensor(d, v, v), tensor(v, d, v), tensor(v, v, d)], -1),
            torch.einsum("g,h,i->ihg", w, w, w).reshape(27))


_V = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _isochoric(law, c, F, J):
    """Cauchy stress and spatial tangent of the isochoric energy: F [.., 3, 3]."""
    I = torch.eye(3, dtype=torch.float64, device=F.device)
    Fb = F * J[..., None, None] ** (-1.0 / 3.0)
    Cb = Fb.transpose(-1, -2) @ Fb
    II = torch.einsum("ij,kl->ijkl", I, I)
    sym = 0.5 * (torch.einsum("ik,jl->ijkl", I, I) + torch.einsum("il,jk->ijkl", I, I))
    if law == "mr":
        tr = Cb.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
        S = 2.0 * (c[0] + tr * c[1]) * I - 2.0 * c[1] * Cb
        D = (4.0 * c[1] * (II - sym)).expand(*F.shape[:-2], 3, 3, 3, 3)
    else:
        b = torch.tensor([2 * c[1], 2 * c[2], 2 * c[2], c[3], c[3], c[2]], dtype=torch.float64, device=F.device)
        E = torch.stack([0.5 * (Cb[..., i, i] - 1.0) if i == j else Cb[..., i, j] for i, j in _V], -1)
        q = b * E
        t = (0.5 * c[0] * torch.exp(0.5 * (E * q).sum(-1)))[..., None]
        at = [[next(k for k, v in enumerate(_V) if set(v) == {i, j}) for j in range(3)] for i in range(3)]
        at = torch.tensor(at, device=F.device)
        S = (t * q)[..., at]
        V = t[..., None] * (q[..., :, None] * q[..., None, :] + torch.diag(b))
        D = V[..., at[:, :, None, None], at[None, None, :, :]]
    s = Fb @ S @ Fb.transpose(-1, -2) / J[..., None, None]
    for k in range(4):  # push one index forward at a time
        D = torch.einsum("...ia,...abcd->...bcdi", Fb, D)
    D = D / J[..., None, None, None, None]
    trs = s.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
    dev = s - trs / 3.0 * I
    P = sym - II / 3.0
    D = torch.einsum("ijab,...abcd,cdkl->...ijkl", P, D, P) + (2.0 / 3.0) * trs[..., None, None] * P
    D = D - (2.0 / 3.0) * (torch.einsum("ij,...kl->...ijkl", I, dev) + torch.einsum("...ij,kl->...ijkl", dev, I))
    return dev, D, I, II, sym


def _faces(m, n):
    """(elements, face nodes, normal direction, side) of the box's loaded boundary faces."""
    ex, ey, ez = m["dims"]
    e = np.arange(ex * ey * ez).reshape(ez, ey, ex)
    a = np.arange(n ** 3).reshape(n, n, n)  # [xi3][xi2][xi1]
    for ni in range(3):
        for side in (0, 1):
            ax = 2 - ni
            if m["surf"][ni].any():
                yield np.take(e, -side, ax).ravel(), np.take(a, -side, ax).ravel(), ni, side


def _elements(m, x, lo, hi, jacobian):
    """Element residuals [e, rows] and Jacobians [e, rows, rows] of elements lo..hi."""
    n, law = m["nxi"], m["law"]
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    N, dN, w = _basis(n)
    nu, npe = m["X"].shape[1], n ** 3
    en = f(m["elem_u"][lo:hi].astype(np.int64))
    z = x[:3 * nu].view(3, nu)[:, en]      # [3, e, a]
    X = f(m["X"])[:, en]
    dz, dX = (torch.einsum("cea,gak->egck", v, dN) for v in (z, X))
    if m["elem_p"] is None:
        psi = torch.ones(27, 1, dtype=torch.float64, device=DEV)
        p = x[3 * nu + lo:3 * nu + hi][:, None].expand(-1, 27)
    else:
        psi = _basis(2)[0]
        p = torch.einsum("gq,eq->eg", psi, x[3 * nu:][f(m["elem_p"][lo:hi].astype(np.int64))])
    Jz, Jx = torch.linalg.det(dz), torch.linalg.det(dX)
    if m["fibre"] is None:  # the material axes are the coordinate axes
        F = dz @ torch.linalg.inv(dX)
    else:
        ang = torch.einsum("cea,ga->egc", f(m["fibre"])[:, en], N)
        t1, t2 = dX[..., 0], dX[..., 1]
        h = torch.linalg.cross(t1, t2)
        R = torch.stack([v / v.norm(dim=-1, keepdim=True) for v in (t1, torch.linalg.cross(h, t1), h)], -1)
        o, u = torch.zeros_like(ang[..., 0]), torch.ones_like(ang[..., 0])
        c, s = torch.cos(ang), torch.sin(ang)
        rot = lambda *r: torch.stack(r, -1).unflatten(-1, (3, 3))  # noqa: E731
        R = R @ rot(c[..., 0], -s[..., 0], o, s[..., 0], c[..., 0], o, o, o, u)
        R = R @ rot(c[..., 1], o, s[..., 1], o, u, o, -s[..., 1], o, c[..., 1])
        R = R @ rot(u, o, o, o, c[..., 2], -s[..., 2], o, s[..., 2], c[..., 2])
        F = dz @ torch.linalg.inv(R.transpose(-1, -2) @ dX)
    J = Jz / Jx
    dev, D, I, II, sym = _isochoric(law, [float(v) for v in m["materials"]], F, J)
    sig = dev + p[..., None, None] * I
    D = D + p[..., None, None, None, None] * (II - 2.0 * sym)
    G = torch.einsum("gak,egki->egai", dN, torch.linalg.inv(dz))  # dN/dz
    jw, xw = Jz * w, Jx * w
    ne, n_p = hi - lo, psi.shape[1]
    r = torch.cat([torch.einsum("eg,egai,egim->ema", jw, G, sig).reshape(ne, 3 * npe),
                   torch.einsum("eg,gq->eq", xw * (J - 1.0), psi)], 1)
    K = None
    if jacobian:
        A = D + torch.einsum("mn,egij->egimjn", I, sig)  # [i, m, j, n]
        T = torch.einsum("eg,egimjn,egbj->emginb", jw, A, G).reshape(ne, 3, 81, 3 * npe)
        B = G.permute(0, 2, 1, 3).reshape(ne, 1, npe, 81)
        K = torch.zeros(ne, 3 * npe + n_p, 3 * npe + n_p, dtype=torch.float64, device=DEV)
        K[:, :3 * npe, :3 * npe] = (B @ T).reshape(ne, 3 * npe, 3 * npe)
        C = torch.einsum("eg,gq,egbn->eqnb", jw, psi, G).reshape(ne, n_p, 3 * npe)
        K[:, 3 * npe:, :3 * npe] = C
        K[:, :3 * npe, 3 * npe:] = C.transpose(1, 2)
    if m["surf"] is not None:
        _surface(m, z, lo, hi, r, K)
    return r, K


def _surface(m, z, lo, hi, r, K):
    """Adds the follower pressure on the loaded faces to r and the off-diagonal blocks of K."""
    n = m["nxi"]
    npe = n ** 3
    t = torch.tensor([0.5 - math.sqrt(0.15), 0.5, 0.5 + math.sqrt(0.15)], dtype=torch.float64, device=DEV)
    w1 = torch.tensor([5.0, 8.0, 5.0], dtype=torch.float64, device=DEV) / 18.0
    v, d = _lagrange(n, t)
    face = lambda a, b: torch.einsum("ga,hb->hgba", a, b).reshape(9, n * n)  # noqa: E731
    N, dN, w = face(v, v), (face(d, v), face(v, d)), torch.einsum("g,h->hg", w1, w1).reshape(9)
    for els, fn, ni, side in _faces(m, n):
        els = els[(els >= lo) & (els < hi)]
        if not len(els):
            continue
        e = torch.from_numpy(els - lo).to(DEV)
        a = torch.from_numpy(fn).to(DEV)
        p = torch.from_numpy(m["surf"][ni][m["elem_u"][els][:, fn]]).to(DEV) @ N.T
        zf = z[:, e][:, :, a]
        g = torch.stack([torch.einsum("cef,gf->egc", zf, q) for q in dN], -1)  # [e, g, c, 2]
        nrm = torch.linalg.cross(g[..., 0], g[..., 1])
        dual = g @ torch.linalg.inv(g.transpose(-1, -2) @ g)
        pw = w * p * ((1 if side else -1) * (-1 if ni == 1 else 1))
        for c in range(3):
            r[e[:, None], c * npe + a] += torch.einsum("eg,eg,gf->ef", pw, nrm[..., c], N)
        if K is None:
            continue
        for q in range(3):
            for s in range(q):
                W = [(nrm[..., q] * dual[..., s, i] - dual[..., q, i] * nrm[..., s]) * pw for i in range(2)]
                k = sum(torch.einsum("eg,gm,gn->emn", W[i], N, dN[i]) for i in range(2))
                row, col = q * npe + a, s * npe + a
                K[e[:, None, None], row[:, None], col[None, :]] += k
                K[e[:, None, None], col[:, None], row[None, :]] += k.transpose(1, 2)


def _dofs(m, lo, hi):
    nu, ne = m["X"].shape[1], len(m["elem_u"])
    en = m["elem_u"][lo:hi].astype(np.int64)
    p = np.arange(lo, hi)[:, None] if m["elem_p"] is None else m["elem_p"][lo:hi].astype(np.int64)
    nd = 3 * nu + (ne if m["elem_p"] is None else int(m["elem_p"].max()) + 1)
    return torch.from_numpy(np.concatenate([en, nu + en, 2 * nu + en, 3 * nu + p], 1)).to(DEV), nd


def _chunks(m):
    ne = len(m["elem_u"])
    return [(i, min(ne, i + 1024)) for i in range(0, ne, 1024)]


def _assemble(m, x, jacobian):
    """(CSR values in pattern order, row of every entry, column, residual); the first three None without a Jacobian."""
    parts = [_dofs(m, lo, hi) for lo, hi in _chunks(m)]
    nd = parts[0][1]
    r = torch.zeros(nd, dtype=torch.float64, device=DEV)
    keys = vals = None
    if jacobian:
        keys = torch.unique(torch.cat([torch.unique((d[:, :, None] * nd + d[:, None, :]).reshape(-1)) for d, _ in parts]))
        vals = torch.zeros(len(keys), dtype=torch.float64, device=DEV)
    for (lo, hi), (d, _) in zip(_chunks(m), parts):
        re, K = _elements(m, x, lo, hi, jacobian)
        r.index_add_(0, d.reshape(-1), re.reshape(-1))
        if jacobian:
            at = torch.searchsorted(keys, (d[:, :, None] * nd + d[:, None, :]).reshape(-1))
            vals.index_add_(0, at, K.reshape(-1))
            del K, at
    return (vals, keys // nd, keys % nd, r) if jacobian else (None, None, None, r)


def _exact_mixed(m):
    vals, row, col, r = _assemble(m, torch.from_numpy(m["x"]).to(DEV), True)
    nu3 = 3 * m["X"].shape[1]
    uu = (row < nu3) & (col < nu3)
    return vals[uu], vals[~uu], r


def _exact_newton(m):
    """Newton with dense solves from the same state to the rounding of the residual."""
    x = torch.from_numpy(m["x"]).to(DEV)
    x[torch.from_numpy(m["dofs"]).to(DEV)] = torch.from_numpy(m["values"]).to(DEV)
    free = torch.ones(len(x), dtype=torch.bool, device=DEV)
    free[torch.from_numpy(m["dofs"]).to(DEV)] = False
    for _ in range(12):
        vals, row, col, r = _assemble(m, x, True)
        A = torch.zeros(len(x), len(x), dtype=torch.float64, device=DEV)
        A[row, col] = vals
        dx = torch.linalg.solve(A[free][:, free], -r[free])
        x[free] += dx
        if float(dx.norm()) < 1e-13 * float(x.norm()):
            break
    return x


def _exact_net(t, kind):
    W = [w.double().to(DEV).requires_grad_() for w in t["weights"]]
    at, b = 0, []
    for i, o in zip(WIDTHS[:-1], WIDTHS[1:]):
        b.append(t["bias"][at + i * o:at + i * o + o].double().to(DEV).requires_grad_())
        at += i * o + o
    h = t["x"].double().to(DEV)
    for l in range(len(W)):
        h = h @ W[l].T + b[l]
        h = torch.tanh(h) if l + 1 < len(W) else h
    if kind == "infer":
        return h.detach()
    loss = ((h - t["y"].double().to(DEV)) ** 2).mean()
    flat = lambda v: torch.cat([a.reshape(-1) for pair in v for a in pair])  # noqa: E731
    params = flat(zip(W, b)).detach()
    gs = torch.autograd.grad(loss, W + b)
    grad = flat(zip(gs[:len(W)], gs[len(W):]))
    m = 0.9 * t["m"].double().to(DEV) + 0.1 * grad
    v = 0.999 * t["v"].double().to(DEV) + 0.001 * grad ** 2
    step = STEP + 1
    new = params - LR * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"loss": loss.detach().reshape(1), "grad": grad, "weights": new}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "infer"):
        return _exact_net(_training(case, seed), kind)
    m = _inputs(case, seed)
    if kind == "batch":
        outs = [_exact_mixed(v) for v in m]
        flat = []
        for k in range(3):
            at, total = _places([len(o[k]) for o in outs])
            flat.append(torch.zeros(total, dtype=torch.float64, device=DEV))
            for a, o in zip(at, outs):
                flat[-1][a:a + len(o[k])] = o[k]
        return flat
    if kind == "newton":
        return _exact_newton(m)
    if kind in ("mixed", "mixed_host"):
        return _exact_mixed(m)
    vals, _, _, r = _assemble(m, torch.from_numpy(m["x"]).to(DEV), kind == "fp64")
    return (vals, r) if kind == "fp64" else r
