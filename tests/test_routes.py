"""Routes that a call takes where its usual one does not apply: the coloured
order, streams under capture, no memory for the element records, a GMRES cycle
whose grid barrier gives up."""
import ctypes as C

import numpy as np
import pytest

from cm_gb300 import FiniteElasticityEquationsSet, _lib
from cm_gb300 import mesh as M

pytestmark = pytest.mark.gpu

REL, FLOOR = 1e-12, 1e-13  # FP64 results per entry, as in the oracle parity tests


@pytest.fixture(scope="module")
def torch():
    import torch as _torch
    if not _torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.load()
    return _torch


def box(torch, dims, nxi=3, pressure="node", load=False):
    m = M.regular_box(*dims, lengths=tuple(0.5 * d for d in dims), nxi_u=nxi, pressure=pressure, law=M.MR,
                      materials=(2.0, 6.0), perturb=0.05, seed=2)
    sp = None
    if load:
        sp = np.zeros((3, m.nu))
        i, j, k = m.node_ijk()
        sp[2, k == 0] = 1.2
        sp[0, i == i.max()] = -0.4
    es = FiniteElasticityEquationsSet(m)
    if load:
        es.set_surface_pressure(sp)
    x = M.deformed_state(m, stretch=1.05, shear=0.03, noise=0.02, pressure=-2.0, seed=4)
    return m, es, x, torch.from_numpy(x).cuda(), sp


def close(got, ref, what):
    err = np.abs(got.cpu().numpy() - ref)
    assert (err <= REL * np.abs(ref) + FLOOR * np.abs(ref).max()).all(), (what, err.max())


def last_error():
    buf = C.create_string_buffer(512)
    _lib.load().fe_last_error(buf, 512)
    return buf.value


def test_coloured_order_takes_no_records(torch):
    """In the coloured order the FP64 Jacobian allocates nothing on the device."""
    _, warm, _, xw, _ = box(torch, (2, 2, 2))
    _, es, _, x, _ = box(torch, (12, 12, 12))
    for e in (warm, es):
        e.set_assembly_order("coloured")
    warm.jacobian_evaluate(xw)
    v = torch.empty(es.nnz, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    es.jacobian_evaluate(x, v)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free


def test_no_memory_for_the_records(torch):
    """A first FP64 Jacobian that finds no memory for its records has the bits
    of the coloured order and leaves no error behind; so do later ones, until
    the order is set again."""
    m, es, _, x, _ = box(torch, (12, 12, 12))  # records: 110 MB
    new = lambda: torch.empty(es.nnz, dtype=torch.float64, device="cuda")  # noqa: E731
    v, coloured, staged, r = new(), new(), new(), torch.empty_like(x)
    other = FiniteElasticityEquationsSet(m)
    other.jacobian_evaluate(x, staged, r)
    other.set_assembly_order("coloured")
    other.jacobian_evaluate(x, coloured, r)
    torch.cuda.synchronize()
    assert not torch.equal(staged, coloured)
    torch.cuda.empty_cache()
    error = last_error()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
    es.jacobian_evaluate(x, v, r)
    torch.cuda.synchronize()
    assert torch.equal(v, coloured) and last_error() == error
    del rest
    torch.cuda.empty_cache()
    es.jacobian_evaluate(x, v.fill_(0.0), r)
    assert torch.equal(v, coloured)
    es.set_assembly_order("staged")
    es.jacobian_evaluate(x, v.fill_(0.0), r)
    assert torch.equal(v, staged)


@pytest.mark.parametrize("load", [False, True])
@pytest.mark.parametrize("nxi,pressure", [(2, "element"), (2, "node"), (3, "element"), (3, "node")])
def test_captured_calls(torch, oracle, nxi, pressure, load):
    """The FP64 Jacobian (with and without the residual) and the residual
    recorded into a graph, at a state written after the recording: the
    oracle's values, for the Jacobian the bits of the coloured order, for the
    residual without a surface load those of the direct call."""
    m, es, x, xd, sp = box(torch, (4, 3, 5), nxi, pressure, load)
    P = oracle.Problem(m)
    P.set_surface_pressure(sp)
    rp, col = P.pattern()
    vo, ro = P.assemble(x, rp, col, nthreads=8)
    new = lambda n: torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")  # noqa: E731
    xin, v, v2, r, r2 = torch.empty_like(xd), new(es.nnz), new(es.nnz), new(es.ndofs), new(es.ndofs)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        es.jacobian_evaluate(xin, v, r)
        es.jacobian_evaluate(xin, v2)
        es.residual_evaluate(xin, r2)
    xin.copy_(xd)
    for _ in range(2):
        for t in (v, v2, r, r2):
            t.fill_(float("nan"))
        graph.replay()
        es.check_status(xd)
        close(v, vo, "values")
        close(r, ro, "residual of the Jacobian")
        close(r2, ro, "residual")
        assert torch.equal(v, v2)
    direct = es.residual_evaluate(xd)
    close(direct, ro, "direct residual")
    if not load:
        assert torch.equal(direct, r2)
    es.set_assembly_order("coloured")
    assert torch.equal(es.jacobian_evaluate(xd), v)


@pytest.mark.parametrize("restart,extra_from", [(30, 1), (30, 2), (30, 17), (4, 13), (4, 14), (4, 15), (4, 16), (4, 17)])
def test_gmres_cycle_gives_up(torch, restart, extra_from):
    """A load step in whose one-launch GMRES cycle a barrier gives up -- in its
    first iterations, around the end of a short cycle where the solution and
    the residual are updated, or in none when the cycle has fewer -- converges
    to the state of an undisturbed one; so does the next step of the handle."""
    from cm_gb300 import FEError, newton as N
    m = M.regular_box(3, 2, 2, nxi_u=3, pressure="node", law=M.MR, materials=(2.0, 6.0))
    bc = N.clamped_stretch_shear_conditions(m, 1.05, 0.02)
    x0 = torch.from_numpy(N.initial_state(m)).cuda()

    def step(es):
        x = x0.clone()
        rep = es.newton_load_step(x, bc.dofs, bc.full, ksp_restart=restart, ksp_max_iterations=4000)
        assert rep["converged"] == 1 and rep["residual_norm"] <= 1e-10, rep
        return x

    es = FiniteElasticityEquationsSet(m)
    ref = step(es)
    es.set_newton_barrier_limits(4096, extra_from)
    # converged states agree as in the other Newton tests: a residual norm of
    # 1e-10 over a smallest stiffness of about 1e-2
    x = step(es)
    assert float((x - ref).abs().max()) <= 1e-8
    # a cycle of four iterations has 16 barriers; the other route sums in another order
    assert torch.equal(x, ref) == (extra_from == 17 and restart == 4)
    es.set_newton_barrier_limits(0, 0)
    assert torch.equal(step(es), ref)
    with pytest.raises(FEError):
        es.set_newton_barrier_limits(0, 1)


@pytest.mark.parametrize("nxi,dims", [(2, (14, 13, 13)), (3, (10, 10, 10)), (2, (40, 40, 40))])
def test_gmres_on_many_rows(torch, nxi, dims):
    """Systems beyond the one-launch cycle, with one, two and four row chunks to
    an SM and short and long rows: the first Newton step of a few GMRES
    iterations against the same method in plain torch (FP64, an orthonormal
    basis, least squares).  The two differ by the rounding of sums of 10^5
    terms through a dozen well-conditioned steps."""
    from cm_gb300 import newton as N
    m = M.regular_box(*dims, nxi_u=nxi, pressure="node" if nxi == 3 else "element", law=M.MR, materials=(2.0, 6.0))
    bc = N.clamped_stretch_shear_conditions(m, 1.05, 0.02) if nxi == 3 else N.uniaxial_symmetry_conditions(m, 1.05)
    its = 12
    es = FiniteElasticityEquationsSet(m)
    x = torch.from_numpy(N.initial_state(m)).cuda()
    got = x.clone()
    rep = es.newton_load_step(got, bc.dofs, bc.full, ksp_max_iterations=its, max_iterations=1)
    assert rep["linear_iterations"] == its
    fixed = torch.as_tensor(np.asarray(bc.dofs, dtype=np.int64)).cuda()
    x[fixed] = torch.as_tensor(np.asarray(bc.full, dtype=np.float64)).cuda()
    free = torch.ones_like(x)
    free[fixed] = 0.0
    r = torch.empty_like(x)
    vals = es.jacobian_evaluate(x, r=r)
    rp, col = (torch.from_numpy(a.astype(np.int64)).cuda() for a in es.csr_pattern())
    row = torch.repeat_interleave(torch.arange(es.ndofs, device="cuda"), rp[1:] - rp[:-1])
    A = torch.sparse_csr_tensor(rp, col, vals * free[row] * free[col], size=(es.ndofs, es.ndofs))
    nu3 = 3 * m.nu
    diag = torch.zeros_like(x).index_add_(0, row[row == col], vals[row == col])
    s = torch.zeros_like(x).index_add_(0, row, torch.where(col < nu3, vals * vals * free[col] / diag[col], 0.0))
    minv = free * torch.where(torch.arange(es.ndofs, device="cuda") < nu3, 1.0 / diag, -1.0 / torch.where(s != 0, s, 1.0))
    b = -r * free
    V, H = [b / b.norm()], torch.zeros(its + 1, its, dtype=torch.float64, device="cuda")
    for k in range(its):
        w = A @ (minv * V[k])
        for _ in range(2):
            for j, v in enumerate(V):
                h = v @ w
                H[j, k] += h
                w = w - h * v
        H[k + 1, k] = w.norm()
        V.append(w / H[k + 1, k])
    e = torch.zeros(its + 1, 1, dtype=torch.float64)
    e[0] = float(b.norm())
    y = torch.linalg.lstsq(H.cpu(), e).solution[:, 0].cuda()
    d = minv * sum(c * v for c, v in zip(y, V))
    assert float((got - x - rep["last_lambda"] * d).norm()) <= 1e-9 * float(d.norm())


@pytest.mark.parametrize("widths,rows", [((4, 256, 9), 2070), ((7, 64, 61), 16500), ((3, 256, 256), 12289)])
def test_network_with_many_rows(torch, widths, rows):
    """Layers of so many rows that they take the large tiles, and of one tile
    of rows fewer, against FP64; the bar of the other network tests."""
    from cm_gb300 import warmstart as W
    net = W.MLP(widths, seed=3, device="cuda")
    g = torch.Generator().manual_seed(2)
    net.flat.add_(0.1 * torch.randn(net.flat.shape, generator=g).cuda())
    x = torch.randn(rows, widths[0], generator=g).cuda()
    for n in (rows, rows - 800):
        h = x[:n].double()
        for l, got in enumerate(net.forward(x[:n])[1:]):
            h = h @ net.W(l).double().T + net.b(l).double()
            if l + 1 < net.layers:
                h = torch.tanh(h)
            assert float((got - h).abs().max()) <= 2e-5 * float(h.abs().max())


@pytest.mark.parametrize("widths", [(4, 256, 256, 64), (4, 24, 3), (9, 5)])
def test_inference_with_many_rows(torch, widths):
    """A row's BF16 prediction has the same bits whether it is asked for among
    few rows (a cluster of blocks to 16 of them) or many (a block)."""
    from cm_gb300 import warmstart as W
    net = W.MLP(widths, seed=3, device="cuda")
    x = torch.randn(2051, widths[0], generator=torch.Generator().manual_seed(2)).cuda()
    y = net.infer_bf16(x)
    parts = [net.infer_bf16(x[i:i + 1000]) for i in range(0, len(x), 1000)]
    assert torch.equal(y, torch.cat(parts))
    assert torch.equal(net.infer_bf16(x[:1024]), net.infer_bf16(x[:1025])[:1024])


def test_inference_with_few_columns(torch):
    """Inputs with fewer columns than the network has, down to none, and in
    other types and layouts: the missing ones are zero."""
    from cm_gb300 import warmstart as W
    net = W.MLP((5, 32, 7), seed=3, device="cuda")
    x = torch.randint(-2, 3, (19, 5), generator=torch.Generator().manual_seed(2)).float().cuda()
    for cols in (0, 1, 3, 5):
        full = torch.zeros_like(x)
        full[:, :cols] = x[:, :cols]
        ref = net.infer_bf16(full)
        for given in (x[:, :cols], x[:, :cols].double(), x[:, :cols].int(), x[:, :cols].cpu(), x.T[:cols].T):
            assert torch.equal(net.infer_bf16(given), ref)


def test_clones_of_clones(torch):
    """A clone, a clone of it whose source is gone, and both with materials and
    loads of their own: the bits of sets created from the mesh."""
    m, es, x, xd, sp = box(torch, (4, 3, 5), load=True)
    first = es.clone()
    es.close()
    second = first.clone(materials=(1.0, 3.0))
    second.set_surface_pressure(None)
    third = second.clone()
    first.close()
    for got, mats, load in ((second, (1.0, 3.0), None), (third, (1.0, 3.0), None), (third.clone((2.0, 6.0)), (2.0, 6.0), sp)):
        ref = FiniteElasticityEquationsSet(m)
        ref.set_materials(mats)
        for e in (got, ref):
            e.set_surface_pressure(load)
        a, b = torch.empty_like(xd), torch.empty_like(xd)
        assert torch.equal(got.residual_evaluate(xd), ref.residual_evaluate(xd))
        assert torch.equal(got.jacobian_evaluate(xd, r=a), ref.jacobian_evaluate(xd, r=b)) and torch.equal(a, b)
        for s, t in zip(got.jacobian_evaluate_mixed(xd, r=a), ref.jacobian_evaluate_mixed(xd, r=b)):
            assert torch.equal(s, t)
        assert torch.equal(a, b)
        assert all(np.array_equal(s, t) for s, t in zip(got.csr_pattern(), ref.csr_pattern()))
        ra = got.element_residuals(xd)
        assert torch.equal(ra, ref.element_residuals(xd))
