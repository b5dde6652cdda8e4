"""The launch shapes of the fused kernels, the row gathers, the GMRES cycle and
the network kernels at the edges of their ranges: one element, the largest mesh
a small-mesh shape takes and the next size up, remainders of the groups and
tiles.

Tolerances: FP64 results per entry as in the oracle parity tests (1e-12
relative, 1e-13 of the largest entry: rounding of sums of at most a few hundred
terms, for elements of equal edges whose strains are a few per cent); the FP32 displacement block 1e-5 of the largest entry (about 60 FP32
roundings of terms of that size in a sum-factorised entry, summed over at most
12 elements); converged Newton states 1e-8 (a residual norm of 1e-10 over a
smallest stiffness of about 1e-2); network values as in the warm-start tests
(2e-5 in FP32, 2e-2 with 8-bit mantissas).
"""
import dataclasses

import numpy as np
import pytest

from cm_gb300 import EquationsSetBatch, FiniteElasticityEquationsSet, _lib
from cm_gb300 import mesh as M
from cm_gb300 import newton as N

pytestmark = pytest.mark.gpu

REL, FLOOR, UU = 1e-12, 1e-13, 1e-5


@pytest.fixture(scope="module")
def torch():
    import torch as _torch
    if not _torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.load()
    return _torch


def check_all(torch, oracle, m, **state):
    """FP64 and mixed assembly and the residual of m against the oracle."""
    x = M.deformed_state(m, **{**dict(stretch=1.05, shear=0.03, noise=0.02, pressure=-2.0, seed=4), **state})
    es = FiniteElasticityEquationsSet(m)
    P = oracle.Problem(m)
    rp, col = P.pattern()
    vo, ro = P.assemble(x, rp, col, nthreads=8)
    xd = torch.from_numpy(x).cuda()
    r, rm = torch.empty_like(xd), torch.empty_like(xd)
    v = es.jacobian_evaluate(xd, r=r)
    r2 = es.residual_evaluate(xd)
    vu, vc = es.jacobian_evaluate_mixed(xd, r=rm)
    es.check_status(xd)

    def close(got, ref, what):
        err = np.abs(got.cpu().numpy() - ref)
        assert (err <= REL * np.abs(ref) + FLOOR * np.abs(ref).max()).all(), (what, err.max())

    close(v, vo, "values")
    for name, got in (("residual", r2), ("residual of the Jacobian", r), ("residual of the mixed assembly", rm)):
        close(got, ro, name)
    full = es.mixed_to_full(vu.cpu().numpy(), vc.cpu().numpy())
    uu_rp, _ = es.mixed_layout()
    is_uu = np.zeros(es.nnz, dtype=bool)
    for i in range(3 * m.nu):
        is_uu[rp[i] - 1:rp[i] - 1 + uu_rp[i + 1] - uu_rp[i]] = True
    S = np.abs(vo).max()
    err = np.abs(full - vo)
    assert (err[~is_uu] <= REL * np.abs(vo[~is_uu]) + FLOOR * S).all(), err[~is_uu].max()
    assert err[is_uu].max() <= UU * S, err[is_uu].max() / S


# Small-mesh shapes end at 2, 3, 4 or 10 elements per SM (304, 456, 608 and
# 1520 on 152 SMs): sizes on both sides of each.
@pytest.mark.parametrize("nxi,dims,pressure", [
    (3, (1, 1, 1), "node"), (3, (1, 1, 1), "element"), (3, (8, 8, 7), "element"), (3, (19, 8, 3), "node"),
    (3, (17, 9, 3), "node"), (3, (19, 8, 4), "element"), (3, (29, 7, 3), "node"),
    (2, (1, 1, 1), "node"), (2, (19, 8, 2), "element"), (2, (61, 5, 1), "node"), (2, (19, 16, 5), "node"),
    (2, (39, 13, 3), "element"),
])
def test_fused_shapes(torch, oracle, nxi, dims, pressure):
    check_all(torch, oracle, M.regular_box(*dims, lengths=tuple(0.5 * d for d in dims), nxi_u=nxi, pressure=pressure,
                                           law=M.MR, materials=(2.0, 6.0), perturb=0.05, seed=2))


@pytest.mark.parametrize("sectors", [5, 12])
@pytest.mark.parametrize("pressure", ["node", "element"])
def test_gather_of_a_fan(torch, oracle, sectors, pressure):
    """Hexahedra around a common edge: rows with more incidences than a
    gathering step (four) or the read-ahead list (eight) holds."""
    m = M.regular_box(sectors, 1, 1, nxi_u=2, pressure=pressure, law=M.MR, materials=(2.0, 6.0))
    t = 2 * np.pi * np.arange(2 * sectors) / (2 * sectors)
    rad = np.where(np.arange(2 * sectors) % 2, 1.4, 1.0)  # ring nodes, between them the far corners
    plane = np.concatenate([[[0.0], [0.0]], [rad * np.cos(t), rad * np.sin(t)]], axis=1)
    per = plane.shape[1]
    X = np.concatenate([np.vstack([plane, np.full((1, per), z)]) for z in (0.0, 0.8)], axis=1)
    quad = np.array([[0, 1 + 2 * i, 1 + (2 * i + 2) % (2 * sectors), 2 + 2 * i] for i in range(sectors)])
    elems = np.ascontiguousarray(np.hstack([quad, quad + per]).astype(np.int32))
    m = dataclasses.replace(m, elem_u=elems, elem_p=elems if pressure == "node" else None, X=np.ascontiguousarray(X))
    check_all(torch, oracle, m, stretch=1.03, noise=0.005)


@pytest.mark.parametrize("members", [1, 9, 17])
def test_batch_members_on_several_streams(torch, members):
    """The per-member launches, more members than streams, one equations set
    twice: each member's outputs are those of its own call, bit for bit,
    directly and from a captured graph."""
    ms = [M.regular_box(2 + i % 3, 2, 1 + i % 2, nxi_u=3 - i % 2, pressure="node" if i % 3 else "element", law=M.MR,
                        materials=(1.0 + i, 3.0)) for i in range(members)]
    sets = [FiniteElasticityEquationsSet(m) for m in ms]
    sets.append(sets[0])
    ms.append(ms[0])
    xs = [torch.from_numpy(M.deformed_state(m, stretch=1.04, noise=0.02, seed=i)).cuda() for i, m in enumerate(ms)]
    refs = []
    for s, x in zip(sets, xs):
        r = torch.empty_like(x)
        u, c = s.jacobian_evaluate_mixed(x, r=r)
        refs += [t.clone() for t in (u, c, r)]
    batch = EquationsSetBatch(sets)
    batch.set_config(5, 1, 1)
    vus, vcs, rs = batch.allocate("cuda")
    got = [t for k in range(len(ms)) for t in (vus[k], vcs[k], rs[k])]

    def same():
        batch.check(xs[0])
        return all(torch.equal(a, b) for a, b in zip(got, refs))

    batch.jacobian_evaluate_mixed(xs, vus, vcs, rs)
    assert same()
    batch.capture(xs, vus, vcs, rs)
    for t in got:
        t.fill_(float("nan"))
    batch.replay(xs[0])
    assert same()


def _newton(torch, m, **options):
    bc = (N.clamped_stretch_shear_conditions(m, 1.05, 0.02) if m.nxi_u == 3 else N.uniaxial_symmetry_conditions(m, 1.05))
    es = FiniteElasticityEquationsSet(m)
    x = torch.from_numpy(N.initial_state(m)).cuda()
    rep = es.newton_load_step(x, bc.dofs, bc.full, **options)
    assert rep["converged"] == 1 and rep["residual_norm"] <= 1e-10, rep
    r = es.residual_evaluate(x)
    r[torch.as_tensor(np.asarray(bc.dofs, dtype=np.int64)).cuda()] = 0.0
    assert abs(float(r.norm()) - rep["residual_norm"]) <= 1e-12
    return x


@pytest.mark.parametrize("nxi,dims,restarts", [
    (2, (1, 1, 2), (30, 45)),      # rows for three blocks; cycles longer than the system
    (3, (3, 2, 2), (15, 30, 200)),  # odd and even restart lengths, the longest
    (3, (7, 7, 6), (30, 200)),     # 9,223 rows, near the most the blocks hold; at 200 not all matrix entries fit
])
def test_gmres_cycle(torch, nxi, dims, restarts):
    m = M.regular_box(*dims, nxi_u=nxi, pressure="node" if nxi == 3 else "element", law=M.MR, materials=(2.0, 6.0))
    xs = [_newton(torch, m, ksp_restart=k, ksp_max_iterations=4000) for k in restarts]
    for x in xs[1:]:
        assert float((x - xs[0]).abs().max()) <= 1e-8


def test_gmres_on_more_rows_than_the_cycle_takes(torch):
    _newton(torch, M.regular_box(8, 8, 7, nxi_u=3, pressure="node", law=M.MR, materials=(2.0, 6.0)),
            ksp_max_iterations=4000)


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("widths,rows", [((1, 1), 1), ((3, 5, 7, 2), 33), ((4, 300, 33, 65), 100), ((5, 64, 64), 257)])
def test_network_shapes(torch, widths, rows):
    """Widths that are no multiple of a tile or of a 16-byte load, one row, and
    rows past a tile: training step and BF16 inference."""
    import mlp_oracle as O
    from cm_gb300 import warmstart as W
    net = W.MLP(widths, seed=3, device="cuda")
    rng = np.random.default_rng(6)
    x = rng.normal(size=(rows, widths[0])).astype(np.float32)
    t = rng.normal(size=(rows, widths[-1])).astype(np.float32)
    params = [(net.W(l).cpu().numpy().astype(np.float64), net.b(l).cpu().numpy().astype(np.float64))
              for l in range(net.layers)]
    hs = O.forward(params, x.astype(np.float64))
    loss_o, dy = O.mse(hs[-1], t.astype(np.float64))
    grads = O.backward(params, hs, dy)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss = net.loss_and_grad(xd, td)
    assert abs(float(loss) - loss_o) <= 2e-5 * loss_o
    for l in range(net.layers):
        assert _rel(net.W(l, net.grad).cpu().numpy(), grads[l][0]) <= 2e-5
        assert _rel(net.b(l, net.grad).cpu().numpy(), grads[l][1]) <= 2e-5
    for a, b in zip(net.forward(xd)[1:], hs[1:]):
        assert _rel(a.cpu().numpy(), b) <= 2e-5
    if max(widths) <= 256:  # the widest layer it takes
        assert _rel(net.infer_bf16(xd).cpu().numpy(), hs[-1]) <= 2e-2


@pytest.mark.parametrize("widths,rows", [((4, 64, 33, 5), 40), ((3, 2), 1)])
def test_training_step_under_capture(torch, widths, rows):
    """A recorded training step (its kernels start before their predecessors
    have ended) gives the bits of the direct one, and steps in a row those of
    steps with a wait after each call."""
    from cm_gb300 import warmstart as W
    g = torch.Generator().manual_seed(1)
    x, y = torch.randn(rows, widths[0], generator=g).cuda(), torch.randn(rows, widths[-1], generator=g).cuda()
    nets = [W.MLP(widths, seed=3, device="cuda") for _ in range(3)]

    def step(net, wait):
        loss = net.loss_and_grad(x, y)
        if wait:
            torch.cuda.synchronize()
        net.adam_step(1e-2)
        if wait:
            torch.cuda.synchronize()
        return loss

    losses = [step(nets[0], True) for _ in range(20)]
    assert all(torch.equal(a, b) for a, b in zip(losses, [step(nets[1], False) for _ in range(20)]))
    assert torch.equal(nets[0].flat, nets[1].flat)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        loss = step(nets[2], False)
    graph.replay()
    assert torch.equal(loss, losses[0])
    one = W.MLP(widths, seed=3, device="cuda")
    step(one, True)
    assert torch.equal(nets[2].flat, one.flat) and torch.equal(nets[2].grad, one.grad)
