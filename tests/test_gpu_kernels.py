"""Kernels and dispatch branches at the sizes where they can go wrong: edges
of tiles and lane groups, remainders, the smallest and largest of a range,
against the general path or an FP64 reference."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import redbirdpy_b200 as rbb  # noqa: E402
from redbirdpy_b200 import engine  # noqa: E402
from redbirdpy_b200.meshgen import kuhn_box  # noqa: E402


def _mesh(cells=(5, 4, 3), h=2.0, seed=0, omega=0.0):
    """A prepared cfg of a box with displaced interior nodes."""
    rng = np.random.default_rng(seed)
    size = np.array(cells) * h
    node, elem = kuhn_box(size, h)
    inside = np.all((node > 0.5 * h) & (node < size - 0.5 * h), axis=1)
    node[inside] += rng.uniform(-0.12, 0.12, (int(inside.sum()), 3)) * h
    nn = node.shape[0]
    prop = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                            np.full(nn, 1.37)])
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=size[None] * [0.4, 0.4, 0], srcdir=np.array([[0, 0, 1.0]]),
               detpos=size[None] * [0.6, 0.6, 0], detdir=np.array([[0, 0, 1.0]]), omega=omega)
    return rbb.meshprep(cfg)[0]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ns", [1, 2, 3, 4, 5, 8, 9, 31, 64])
def test_tet_gradient_equals_summed_jacobian_rows(ns, cplx):
    """rb_jac_grad = the column sums of rb_jac's rows over the pairs
    (s, lam_s), which go through another kernel.  Both are FP64 sums of about
    24 x 16 x ns products per node; 1e-13 of the largest sum of magnitudes
    allows each some hundred rounding errors."""
    mesh = engine.mesh_of(_mesh())
    g = torch.Generator("cuda").manual_seed(ns)
    dt = torch.complex128 if cplx else torch.float64
    phi = torch.randn((mesh.nn, ns + 3), generator=g, device="cuda", dtype=dt)
    lam = torch.randn((mesh.nn, ns), generator=g, device="cuda", dtype=dt)
    got = engine.jacobian_grad(mesh, phi, lam, ns)
    pairs = np.column_stack([np.arange(ns), ns + np.arange(ns), np.ones(ns)])
    fields = torch.cat([phi[:, :ns], lam], 1).contiguous()
    for g_, what in zip(got, ("mua_nodal", "D")):
        J = engine.jacobian(mesh, fields, pairs, what, out_dtype=torch.float64)
        J = J.real if cplx else J
        scale = J.abs().sum(0).max()
        assert (g_ - J.sum(0)).abs().max() <= 1e-13 * 16 * scale, what
    only = engine.jacobian_grad(mesh, phi, lam, ns, True, False)
    assert only[1] is None and torch.equal(only[0], got[0])


def _system(n, cplx, seed, dense_row=False):
    """A random sparse symmetric (complex: with a positive imaginary part),
    diagonally dominant matrix, optionally with one full row and column."""
    from scipy import sparse

    rng = np.random.default_rng(seed)
    i = rng.integers(0, n, 5 * n)
    j = np.clip(i + rng.integers(-40, 41, 5 * n), 0, n - 1)
    v = rng.uniform(-1, 0, 5 * n) * (1 + (0.2j if cplx else 0))
    A = sparse.coo_matrix((v, (i, j)), shape=(n, n)).tocsr()
    A = A + A.T
    if dense_row:
        r = sparse.coo_matrix((np.full(n, -1e-3), (np.full(n, n // 2), np.arange(n))), shape=(n, n)).tocsr()
        A = A + r + r.T
    d = np.asarray(abs(A).sum(1)).ravel() + rng.uniform(0.05, 0.1, n)
    return (A + sparse.diags(d * (1 + (0.1j if cplx else 0)))).tocsr()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,k,dense_row", [(1, 1, False), (5, 3, False), (33, 2, True), (2047, 5, False),
                                           (2049, 1, False), (4097, 9, True), (8193, 37, False), (16385, 2, False),
                                           (32767, 3, False)])
def test_one_launch_solve_of_small_systems(n, k, dense_row, cplx):
    """The one-launch solve at the edges of its layouts (fewer rows than
    blocks, one row past a thread's share, a row too long for its slice, odd
    column counts, a zero column) against SuperLU and the separate kernels.
    Both refine to the FP64 floor of well-conditioned systems (condition
    below 1e3): 1e-11 of the largest entry."""
    from scipy.sparse.linalg import splu

    A = _system(n, cplx, n + k, dense_row)
    rng = np.random.default_rng(1)
    B = rng.standard_normal((n, k))
    if k > 1:
        B[:, k // 2] = 0.0
    mat = engine.DeviceMatrix.from_scipy(A)
    Bd = torch.as_tensor(B, device="cuda")
    X, info = engine.solve(mat, Bd)
    assert info["flag"] == 0 and info["launches"] == 2, info
    ref = splu(A.tocsc()).solve(B.astype(A.dtype))
    scale = np.abs(ref).max()
    assert np.abs(X.cpu().numpy() - ref).max() <= 1e-11 * scale
    if k > 1:
        assert not X[:, k // 2].any()
    X2, info2 = engine.solve(mat, Bd, profile=True)
    assert info2["flag"] == 0 and info2["launches"] > 2
    assert (X - X2).abs().max() <= 1e-11 * scale
    X3, info3 = engine.solve(mat, Bd, x0=X)  # from the solution
    assert info3["flag"] == 0 and info3["launches"] == 2
    assert (X3 - X).abs().max() <= 1e-11 * scale


def test_one_launch_solve_reports_failure():
    """A capped solve ends unconverged (flag 1), a non-finite column is
    flagged (2) while the others still solve."""
    A = _system(700, False, 3)
    mat = engine.DeviceMatrix.from_scipy(A)
    B = torch.randn((700, 4), device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(2))
    _, info = engine.solve(mat, B, maxiter=1, max_outer=1)
    assert info["flag"] == 1 and info["launches"] == 2
    good, _ = engine.solve(mat, B)
    B2 = B.clone()
    B2[5, 1] = float("nan")
    X, info = engine.solve(mat, B2)
    assert info["flag"] == 2
    keep = [0, 2, 3]
    assert (X[:, keep] - good[:, keep]).abs().max() <= 1e-12 * good.abs().max()


def _box_cfg(cells, h, omega, ns, nd, seed=0, hole=False):
    """A prepared box with nodal properties (a 4x mua / 3x mus inclusion) and
    random optodes inside; ``hole`` leaves out a ball of tets, so that groups
    and aggregates are partly empty."""
    rng = np.random.default_rng(seed)
    size = np.array(cells) * h
    node, elem = kuhn_box(size, h)
    inside = np.all((node > 0.5 * h) & (node < size - 0.5 * h), axis=1)
    node[inside] += rng.uniform(-0.12, 0.12, (int(inside.sum()), 3)) * h
    if hole:
        c = node[elem - 1].mean(axis=1)
        elem = elem[np.linalg.norm(c - size * [0.3, 0.3, 0.3], axis=1) > 0.2 * size.min()]
        used = np.unique(elem)
        remap = np.zeros(node.shape[0] + 1, dtype=np.int64)
        remap[used] = np.arange(1, used.size + 1)
        node, elem = node[used - 1], remap[elem]
    nn = node.shape[0]
    prop = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                            np.full(nn, 1.37)])
    inc = np.linalg.norm(node - size * [0.6, 0.5, 0.4], axis=1) < 0.15 * size.min()
    prop[inc, :2] *= [4, 3]
    pts = rng.uniform(0.55, 0.9, (ns + nd, 3)) * size * [1, 1, 0]
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=pts[:ns], srcdir=np.array([[0, 0, 1.0]]), detpos=pts[ns:],
               detdir=np.array([[0, 0, 1.0]]), omega=omega)
    return rbb.meshprep(cfg)[0]


@pytest.mark.parametrize("omega", [0.0, 2 * np.pi * 1e8])
@pytest.mark.parametrize("cells,cols,hole", [((28, 27, 25), (1, 2), True), ((28, 27, 25), (17, 20), True),
                                             ((40, 24, 20), (31, 33), False), ((28, 27, 25), (33, 34), False),
                                             ((27, 28, 26), (64, 64), True), ((28, 27, 25), (70, 61), False)])
def test_vcycle_solve_matches_the_two_level_form(cells, cols, hole, omega, monkeypatch):
    """The three-level cycle at lane layouts from 4 to 128 columns (padded
    counts, both column slices of complex solves, more than one block of 128)
    on meshes with partly empty groups: the solution of the two-level and
    Jacobi-only forms, each refined to the FP64 floor (the bars of the
    two-level form's own tests: phi 1e-9, detectors 1e-6), in fewer
    iterations, and again from a perturbed start."""
    from redbirdpy_b200.forward import forward_device

    monkeypatch.setattr(engine, "VCYCLE_ENTRIES", 0)  # few columns too
    cfg = _box_cfg(cells, 1.5, omega, *cols, hole=hole)
    d1, p1, _, mat, i1 = forward_device(cfg)
    assert mat.n >= engine.COARSE_MIN_NODES and engine.mesh_of(cfg).mid_level() is not None
    assert i1["flag"] == 0 and i1["relres"] <= 1e-12 and i1["coarse_nc"] > 0
    d0, p0, _, _, i0 = forward_device(cfg, coarse=True)
    assert i0["flag"] == 0 and i1["iters"] < 0.7 * i0["iters"], (i1["iters"], i0["iters"])
    assert (p1 - p0).abs().max() <= 1e-9 * p0.abs().max()
    assert ((d1 - d0).abs() / d0.abs()).max() <= 1e-6
    _, p2, _, _, i2 = forward_device(cfg, x0=p1 * (1 + 1e-3))
    assert i2["flag"] == 0 and (p2 - p0).abs().max() <= 1e-9 * p0.abs().max()


def test_vcycle_zero_and_non_finite_columns(monkeypatch):
    """A zero column stays exactly zero; a non-finite one is flagged and the
    others still solve (through the two-level form)."""
    monkeypatch.setattr(engine, "VCYCLE_ENTRIES", 0)
    cfg = _box_cfg((28, 27, 25), 1.5, 0.0, 3, 2)
    mesh = engine.mesh_of(cfg)
    mat = engine.assemble(mesh, engine.Optics.from_cfg(mesh, cfg))
    B = engine.locate_optodes(mesh, cfg).rhs(mesh)
    B[:, 1] = 0.0
    X, info = engine.solve(mat, B)
    assert info["flag"] == 0 and not X[:, 1].any()
    B2 = B.clone()
    B2[7, 2] = float("inf")
    X2, info2 = engine.solve(mat, B2)
    assert info2["flag"] == 2
    keep = [0, 1, 3, 4]
    assert (X2[:, keep] - X[:, keep]).abs().max() <= 1e-9 * X.abs().max()


def _delaunay_cfg(seed=0):
    """An irregular mesh: rows of more than 16 neighbours."""
    from scipy.spatial import Delaunay

    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(6.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    node = g + rng.uniform(-0.25, 0.25, g.shape)
    elem = Delaunay(node).simplices + 1
    x = node[elem - 1]
    vol = np.abs(np.einsum("ij,ij->i", np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), x[:, 3] - x[:, 0])) / 6
    elem = elem[vol > 1e-6]
    prop = np.tile([0.01, 1.0, 0.0, 1.37], (node.shape[0], 1))
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=np.array([[2.0, 2.0, 0]]), srcdir=np.array([[0, 0, 1.0]]),
               detpos=np.array([[3.0, 3.0, 0]]), detdir=np.array([[0, 0, 1.0]]), omega=0)
    return rbb.meshprep(cfg)[0]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("mesh_kind", ["box", "delaunay"])
@pytest.mark.parametrize("ns,nd", [(4, 4), (12, 8), (4, 64), (64, 4), (28, 36), (64, 64)])
def test_grid_jacobian_rows_equal_the_general_kernels(ns, nd, mesh_kind, cplx, monkeypatch):
    """The pipelined kernel of the FP64-formed FP32 rows (both parameters, and
    node slabs of odd widths) = rb_jac's rows per quantity, bit for bit: the
    same products in the same order."""
    monkeypatch.setattr(engine, "JAC_GRID_NODES", 1)
    mesh = engine.mesh_of(_mesh((7, 5, 4)) if mesh_kind == "box" else _delaunay_cfg())
    assert (mesh.rmax <= 16) == (mesh_kind == "box") and mesh.rmax <= 32 and mesh.emax <= 64
    g = torch.Generator("cuda").manual_seed(ns * 100 + nd)
    dt = torch.complex128 if cplx else torch.float64
    phi = torch.randn((mesh.nn, ns + nd + 1), generator=g, device="cuda", dtype=dt)
    s, d = np.meshgrid(np.arange(ns), ns + np.arange(nd))
    sd = np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)])
    kind = engine._lib.RB_JAC_SPLIT_F32_ACC64 if cplx else engine._lib.RB_JAC_F32_ACC64
    cols, det0, ndet, psrc, pdet, colsd, ps, pd, gnsd = engine._pair_dev(sd, phi.device)
    assert gnsd < 0
    rows = (2 if cplx else 1) * ns * nd
    nn = mesh.nn
    for mode, whats in (("exact", (engine._lib.RB_JAC_MUA_NODAL, engine._lib.RB_JAC_D)),
                        ("reference", (engine._lib.RB_JAC_MUA_REF,))):
        params = ("mua", "D")[: len(whats)]
        J, K = engine.jacobian_matrix(mesh, phi, sd, params, mode, acc64=True)
        ref = torch.full_like(J, float("nan"))
        for p, w in enumerate(whats):
            engine.call("rb_jac", engine.ctypes.byref(mesh.struct), w, engine.ptr(phi),
                        engine._lib.RB_C128 if cplx else engine._lib.RB_F64, phi.shape[1], engine.ptr(colsd),
                        len(cols), det0, ndet, engine.ptr(ps), engine.ptr(pd), gnsd, engine.ptr(ref[:, p * nn:]),
                        ref.shape[1], kind, mesh.rmax, mesh.emax, engine.ptr(mesh.evol), engine.ptr(mesh.ddd),
                        engine.stream())
        assert torch.equal(J[:, :K], ref[:, :K])
        op = engine.SlabJacobian(mesh, phi, sd, params, mode, width=37, acc64=True)
        for a, b in op.ranges():
            Js, ks = op.slab(a, b)
            want = torch.cat([ref[:, p * nn + a:p * nn + b] for p in range(len(whats))], 1)
            assert ks == want.shape[1] and torch.equal(Js[:, :ks], want), (a, b)
    assert rows == J.shape[0]


@pytest.mark.parametrize("M,pad", [(1, 0), (2, 3), (63, 1), (64, 0), (65, 0), (128, 5), (1000, 0), (9473, 0), (9535, 1)])
def test_chol_solve_segments(M, pad):
    """L L^T x = b over block rows handed on between thread blocks: one block
    row, ragged last rows, strided factors, and more block rows than SMs (9473
    = 148 x 64 + 1).  L is unit-diagonal plus a small lower part, so that
    ||L^-1||_inf <= 1 / (1 - 0.5) and the error bound M eps cond is below
    M x 2.2e-16 x 16; with the short workspace and in a captured launch the
    bits are the same."""
    g = torch.Generator("cuda").manual_seed(M)
    ld = M + pad
    L = torch.rand((M, ld), generator=g, device="cuda", dtype=torch.float64).sub_(0.5).mul_(1.0 / M)
    Lt = torch.tril(L[:, :M], -1) + torch.eye(M, device="cuda", dtype=torch.float64)
    H = torch.full((M, ld), float("nan"), device="cuda", dtype=torch.float64)
    H[:, :M] = Lt
    # rb_cholesky leaves each diagonal block's inverse in its strict upper triangle
    for k in range(0, M, 64):
        e = min(M, k + 64)
        X = torch.linalg.inv(Lt[k:e, k:e])
        H[k:e, k:e] = Lt[k:e, k:e] + torch.tril(X, -1).T
    x0 = torch.randn(M, generator=g, device="cuda", dtype=torch.float64)
    b = Lt @ (Lt.T @ x0)
    tol = M * 2.2e-16 * 16 * float(x0.abs().max())
    wb = engine._lib.lib().rb_chol_solve_work_bytes(M)

    def solve(x, w, nbytes):
        engine.call("rb_chol_solve", engine.ptr(H), M, ld, engine.ptr(x), engine.ptr(w), nbytes, engine.stream())

    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    x = b.clone()
    solve(x, work, wb)
    assert float((x - x0).abs().max()) <= tol
    short = torch.empty(M * 8, dtype=torch.uint8, device="cuda")
    xs = b.clone()
    solve(xs, short, M * 8)
    assert torch.equal(x, xs)
    xc = b.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve(xc, work, wb)
    for _ in range(2):
        xc.copy_(b)
        graph.replay()
        assert torch.equal(x, xc)
    with pytest.raises(Exception, match="workspace too small"):
        solve(xs, short, M * 8 - 1)


@pytest.mark.parametrize("M,pad", [(1, 0), (15, 1), (16, 0), (17, 0), (33, 0), (63, 0), (64, 2), (81, 0), (129, 0)])
def test_cholesky_diagonal_block_and_its_inverse(M, pad):
    """The 16-column steps of a diagonal block: factor and inverse (strict
    upper triangle, transposed) at every remainder, a strided matrix, and the
    first pivot that is not positive.  A = B B^T / M + I has condition at most
    1 + 4 (M + 7) / M < 40, so M eps cond < M x 1e-14 bounds both."""
    g = torch.Generator("cuda").manual_seed(M)
    B = torch.randn((M, M + 7), generator=g, device="cuda", dtype=torch.float64)
    A = B @ B.T / (M + 7) + torch.eye(M, device="cuda", dtype=torch.float64)
    ld = M + pad

    def factor(a):
        H = torch.zeros((M, ld), device="cuda", dtype=torch.float64)
        H[:, :M] = a
        work = torch.empty(engine._lib.lib().rb_cholesky_work_bytes(), dtype=torch.uint8, device="cuda")
        engine.call("rb_cholesky", engine.ptr(H), M, ld, engine.ptr(work), work.numel(), engine.stream())
        return H[:, :M]

    H = factor(A)
    L = torch.linalg.cholesky(A)
    assert float((torch.tril(H) - L).abs().max()) <= M * 1e-14 * float(L.abs().max())
    for k in range(0, M, 64):
        e = min(M, k + 64)
        X = torch.linalg.inv(L[k:e, k:e])
        assert float((torch.triu(H[k:e, k:e], 1).T - torch.tril(X, -1)).abs().max()) <= M * 1e-14 * 4
    for p in sorted({0, M // 2, M - 1}):
        bad = A.clone()
        bad[p, p] = -1.0
        with pytest.raises(Exception, match=f"at row {p}$"):
            factor(bad)


def test_pinned_pool_is_bounded_and_thread_safe():
    """A full pool falls back to plain copies, a released buffer makes room
    for another shape, and threads never share a buffer."""
    import threading

    pool = engine.PinnedPool(per_shape=3, min_bytes=0, max_bytes=3 << 20)
    ts = [torch.full((1 << 17,), float(i), device="cuda", dtype=torch.float64) for i in range(4)]
    arrs = [pool.to_numpy(t) for t in ts]  # the fourth finds no room
    assert pool._bytes() == 3 << 20 and all((a == i).all() for i, a in enumerate(arrs))
    b = pool.to_numpy(torch.ones(1 << 18, device="cuda", dtype=torch.float64))
    assert pool._bytes() == 3 << 20 and (b == 1).all()
    del arrs[0], arrs[0]
    c = pool.to_numpy(torch.full((1 << 18,), 7.0, device="cuda", dtype=torch.float64))
    assert pool._bytes() == 3 << 20 and (c == 7).all() and (b == 1).all()
    assert all((a == i + 2).all() for i, a in enumerate(arrs))
    del arrs, c
    pool.trim()
    assert pool._bytes() == 0
    bad = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(20):
                v = float(100 * k + i)
                a = pool.to_numpy(torch.full((64, 64), v, device="cuda", dtype=torch.float64))
                if not (a == v).all():
                    bad.append(v)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad


def test_captured_step_budget_covers_its_jacobi_solves(monkeypatch):
    """A captured step on a mesh whose checked solves take the V-cycle (24
    iterations where Jacobi alone takes 130): its budget is for the solves it
    runs, so it converges; also a batch of such instances."""
    from redbirdpy_b200.adjoint import BatchModel, CapturedStep, DeviceModel, detector_values

    monkeypatch.setattr(engine, "VCYCLE_ENTRIES", 0)
    cfg = _box_cfg((34, 30, 18), 2.0, 0.0, 5, 4)
    cfgs = [_box_cfg(c, 2.0, 0.0, 4, 3) for c in ((24, 20, 12), (20, 24, 14), (28, 20, 10))]
    for model, cs in ((DeviceModel(cfg), [cfg]), (BatchModel(cfgs), cfgs)):
        assert model.mesh.nn >= engine.COARSE_MIN_NODES
        prop = np.vstack([c["prop"] for c in cs])
        mua = torch.as_tensor(prop[:, 0].copy(), device="cuda")
        dco = torch.as_tensor(1.0 / (3.0 * (prop[:, 0] + prop[:, 1])), device="cuda")
        with torch.no_grad():
            ref = detector_values(model, mua, dco)
        step = CapturedStep(model, lambda det: det.square().sum(), mua, dco)
        det = step(mua, dco)[1].detach()
        assert int(torch.as_tensor(step.status).max()) == 0
        assert float((det - ref).abs().max()) <= 1e-10 * float(ref.abs().max())
        step.release()


@pytest.mark.parametrize("omega", [0.0, 2 * np.pi * 1e8])
def test_batch_vcycle_equals_jacobi(omega):
    """Stacked instances of unequal spacing and scale (one with D 1000 times
    smaller, one with fewer optodes, so zero columns): the V-cycle's fields
    against Jacobi's, per instance; statuses; a solve cut short reports every
    instance; a batch of small instances keeps Jacobi alone."""
    from redbirdpy_b200.adjoint import BatchModel

    cfgs = [_box_cfg(c, h, omega, ns, 2) for c, h, ns in
            (((24, 20, 12), 1.0, 3), ((20, 24, 14), 3.0, 5), ((28, 20, 10), 2.0, 1), ((19, 21, 11), 0.5, 5))]
    bm = BatchModel(cfgs)
    assert bm.solve_kw["coarse"] == "blocks" and bm.mesh.layout is not None
    prop = np.vstack([c["prop"] for c in cfgs])
    mua = torch.as_tensor(prop[:, 0].copy(), device="cuda")
    dco = torch.as_tensor(1.0 / (3.0 * (prop[:, 0] + prop[:, 1])), device="cuda")
    dco[int(bm.node_off[1]):int(bm.node_off[2])] *= 1e-3
    mat = engine.assemble(bm.mesh, bm.optics(mua, dco))
    X, info = engine.solve(mat, bm.B, **bm.solve_kw)
    assert info["spmm_kernel"] == "vc_spmm_kernel" and info["flag"] == 0 and not info["inst_status"].any()
    Y, inf2 = engine.solve(mat, bm.B, **dict(bm.solve_kw, coarse=False))
    assert inf2["spmm_kernel"] != "vc_spmm_kernel" and not inf2["inst_status"].any()
    assert info["inst_relres"].shape == (4, bm.B.shape[1]) and info["inst_relres"].max() <= 1e-14
    for a, b in zip(bm.node_slices(X), bm.node_slices(Y)):
        assert float((a - b).abs().max()) <= 1e-10 * float(b.abs().max())
    assert float(X[int(bm.node_off[2]):int(bm.node_off[3]), 1:5].abs().max()) == 0.0
    _, short = engine.solve(mat, bm.B, **dict(bm.solve_kw, maxiter=2, max_outer=1))
    assert short["flag"] == 1 and (short["inst_status"] == 1).all()
    small = BatchModel([_box_cfg((14, 12, 8), 2.0, omega, 3, 2) for _ in range(12)])
    assert small.mesh.nn >= engine.COARSE_MIN_NODES and small.solve_kw["coarse"] is False
    assert small.mesh.layout is None


@pytest.mark.parametrize("cells,ns,nd,cplx,one", [
    ((21, 20, 20), 3, 4, False, True), ((20, 20, 20), 42, 41, False, True), ((20, 20, 20), 43, 42, False, False),
    ((20, 20, 20), 25, 25, True, True), ((20, 20, 20), 26, 26, True, False), ((30, 28, 26), 9, 9, False, True),
    ((30, 28, 26), 9, 10, False, False), ((20, 20, 20), 64, 64, True, False), ((32, 31, 31), 2, 1, True, False)])
def test_solve_routes_between_one_launch_and_vcycle(cells, ns, nd, cplx, one):
    """Both sides of the lines between the one-launch solve and the V-cycle
    (entries, node factor, complex weight, rows of one launch): the route, and the
    fields against the FP64 solve.  Both are refined to a relative residual of
    1e-15, times a condition number below 1e4 times 10."""
    cfg = _box_cfg(cells, 2.0, 2 * np.pi * 1e8 if cplx else 0.0, ns, nd)
    model = rbb.adjoint.DeviceModel(cfg)
    mua = torch.as_tensor(cfg["prop"][:, 0].copy(), device="cuda")
    dco = torch.as_tensor(1.0 / (3.0 * (cfg["prop"][:, 0] + cfg["prop"][:, 1])), device="cuda")
    mat = engine.assemble(model.mesh, model.optics(mua, dco))
    X, info = engine.solve(mat, model.B)
    assert info["flag"] == 0 and (info["launches"] == 2) == one
    assert (info["coarse_nc"] > 0) == (not one)
    Y, _ = engine.solve(mat, model.B, precision="fp64")
    assert float((X - Y).abs().max()) <= 1e-10 * float(Y.abs().max())


@pytest.mark.parametrize("mesh_kind", ["box", "delaunay"])
@pytest.mark.parametrize("cplx,ld,s0,sstep,d0", [
    (False, 40, 0, 1, 12),   # two ranges on 16 bytes: bulk copies
    (False, 40, 1, 1, 14),   # sources start off 16 bytes
    (False, 40, 0, 1, 13),   # detectors start off 16 bytes
    (False, 41, 0, 1, 12),   # rows start off 16 bytes
    (False, 40, 0, 2, 26),   # every other column
    (True, 41, 1, 1, 15),    # complex entries are 16 bytes each
    (True, 41, 0, 2, 26)])
def test_grid_jacobian_rows_by_either_copy(mesh_kind, cplx, ld, s0, sstep, d0, monkeypatch):
    """The fetch by bulk copies and the one by 16- or 8-byte copies, along the
    line between them: rb_jac's rows bit for bit."""
    monkeypatch.setattr(engine, "JAC_GRID_NODES", 1)
    mesh = engine.mesh_of(_mesh((6, 5, 4)) if mesh_kind == "box" else _delaunay_cfg())
    ns, nd = 12, 8
    g = torch.Generator("cuda").manual_seed(ld + d0)
    dt = torch.complex128 if cplx else torch.float64
    phi = torch.randn((mesh.nn, ld), generator=g, device="cuda", dtype=dt)
    s, d = np.meshgrid(s0 + sstep * np.arange(ns), d0 + np.arange(nd))
    sd = np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)])
    J, K = engine.jacobian_matrix(mesh, phi, sd, ("mua",), "exact", acc64=True)
    cols, det0, ndet, psrc, pdet, colsd, ps, pd, gnsd = engine._pair_dev(sd, phi.device)
    assert gnsd < 0
    kind = engine._lib.RB_JAC_SPLIT_F32_ACC64 if cplx else engine._lib.RB_JAC_F32_ACC64
    ref = torch.full_like(J, float("nan"))
    engine.call("rb_jac", engine.ctypes.byref(mesh.struct), engine._lib.RB_JAC_MUA_NODAL, engine.ptr(phi),
                engine._lib.RB_C128 if cplx else engine._lib.RB_F64, ld, engine.ptr(colsd), len(cols), det0, ndet,
                engine.ptr(ps), engine.ptr(pd), gnsd, engine.ptr(ref), ref.shape[1], kind, mesh.rmax, mesh.emax,
                engine.ptr(mesh.evol), None, engine.stream())
    assert torch.equal(J[:, :K], ref[:, :K])


@pytest.mark.parametrize("mesh_kind", ["box", "delaunay"])
@pytest.mark.parametrize("ns,nd,cplx", [(1, 1, False), (2, 3, True), (3, 4, False), (5, 7, False), (5, 7, True),
                                        (11, 13, False), (11, 13, True), (33, 17, False), (33, 17, True),
                                        (63, 61, False), (63, 61, True), (7, 64, False), (7, 64, True)])
def test_grid_jacobian_rows_at_any_counts(ns, nd, cplx, mesh_kind, monkeypatch):
    """Counts that are no multiples of 4 (and tiles too empty for the kernel):
    rb_jac's rows, pair by pair, bit for bit, at an even and an odd row stride
    of the fields."""
    monkeypatch.setattr(engine, "JAC_GRID_NODES", 1)
    mesh = engine.mesh_of(_mesh((6, 5, 4)) if mesh_kind == "box" else _delaunay_cfg())
    dt = torch.complex128 if cplx else torch.float64
    kind = engine._lib.RB_JAC_SPLIT_F32_ACC64 if cplx else engine._lib.RB_JAC_F32_ACC64
    s, d = np.meshgrid(np.arange(ns), ns + np.arange(nd))
    sd = np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)])
    for ld in (ns + nd + (ns + nd) % 2, ns + nd + 1 - (ns + nd) % 2):
        g = torch.Generator("cuda").manual_seed(ld)
        phi = torch.randn((mesh.nn, ld), generator=g, device="cuda", dtype=dt)
        J, K = engine.jacobian_matrix(mesh, phi, sd, ("mua",), "exact", acc64=True)
        cols, det0, ndet, psrc, pdet, colsd, ps, pd, _ = engine._pair_dev(sd, phi.device)
        ref = torch.full_like(J, float("nan"))
        engine.call("rb_jac", engine.ctypes.byref(mesh.struct), engine._lib.RB_JAC_MUA_NODAL, engine.ptr(phi),
                    engine._lib.RB_C128 if cplx else engine._lib.RB_F64, ld, engine.ptr(colsd), len(cols), det0, ndet,
                    engine.ptr(ps), engine.ptr(pd), ns * nd, engine.ptr(ref), ref.shape[1], kind, mesh.rmax, mesh.emax,
                    engine.ptr(mesh.evol), None, engine.stream())
        assert torch.equal(J[:, :K], ref[:, :K]), ld
