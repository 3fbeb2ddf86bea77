"""Which form of the block solve a call takes, and what each form accepts."""

import numpy as np
import pytest
import torch

import redbirdpy_b200 as rbb
from redbirdpy_b200 import _lib, engine
from redbirdpy_b200.meshgen import kuhn_box

pytestmark = pytest.mark.gpu


def _matrix(cells, omega=0.0, seed=0):
    """The device matrix of a homogeneous box (1.5 mm, jittered properties)."""
    rng = np.random.default_rng(seed)
    size = np.array(cells) * 1.5
    node, elem = kuhn_box(size, 1.5)
    nn = node.shape[0]
    prop = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                            np.full(nn, 1.37)])
    pos = size[None] * [[0.4, 0.4, 0.0]]
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=pos, srcdir=np.array([[0, 0, 1.0]]), detpos=pos,
               detdir=np.array([[0, 0, 1.0]]), omega=omega)
    cfg, _ = rbb.meshprep(cfg)
    mesh = engine.mesh_of(cfg)
    return engine.assemble(mesh, engine.Optics.from_cfg(mesh, cfg))


def _rhs(n, k, seed=0):
    g = torch.Generator("cuda").manual_seed(seed)
    B = torch.randn((n, k), generator=g, device="cuda", dtype=torch.float64)
    return B * (torch.rand((n, k), generator=g, device="cuda") < 0.01)


@pytest.mark.parametrize("omega", [0.0, 2 * np.pi * 1e8])
@pytest.mark.parametrize("k", [4, 68])
def test_cycle_solve_of_a_right_hand_side_off_16_bytes(k, omega, monkeypatch):
    """A contiguous view that starts 8 bytes into its storage is solved like
    its copy, bit for bit."""
    monkeypatch.setattr(engine, "VCYCLE_ENTRIES", 0)
    mat = _matrix((28, 27, 25), omega)
    B = _rhs(mat.n, k)
    view = torch.empty(mat.n * k + 1, dtype=torch.float64, device="cuda")[1:].view(mat.n, k)
    view.copy_(B)
    assert view.is_contiguous() and view.data_ptr() % 16 == 8
    X, info = engine.solve(mat, B)
    Y, info2 = engine.solve(mat, view)
    assert info["coarse_nc"] > 0 and info2["coarse_nc"] > 0 and info["flag"] == 0
    assert torch.equal(X, Y)


@pytest.mark.parametrize("cplx", [False, True])
def test_small_solves_of_different_sizes_from_several_threads(cplx):
    """Solves whose plans need different amounts of shared memory, through
    the same kernel, from threads of one process: each its own solution."""
    import threading

    omega = 2 * np.pi * 1e8 if cplx else 0.0
    mats = [_matrix(c, omega) for c in ((4, 4, 3), (9, 8, 7), (12, 11, 10), (15, 14, 13))]
    rhs = [_rhs(m.n, 2, seed=i) for i, m in enumerate(mats)]
    want = [engine.solve(m, b)[0] for m, b in zip(mats, rhs)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(40):
                    X, info = engine.solve(mats[i], rhs[i])
                    if info["flag"] or info["launches"] != 2 or not torch.equal(X, want[i]):
                        bad.append((i, info))
        except Exception as e:  # a refused launch
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(mats))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


@pytest.mark.parametrize("cells,k,cplx,one", [((9, 9, 8), 128, False, True), ((20, 20, 20), 128, False, True),
                                              ((25, 25, 24), 128, False, False), ((25, 25, 24), 128, True, False),
                                              ((25, 25, 24), 8, True, True), ((32, 31, 30), 128, False, False),
                                              ((32, 31, 30), 130, False, False), ((32, 31, 30), 16, False, True)])
def test_wide_solves_leave_the_one_launch_form(cells, k, cplx, one):
    """Jacobi solves whose columns would take many waves of the one launch run
    the separate kernels; row groups asked for are used; every form refines to
    a relative residual of 1e-15 (condition below 1e4: 1e-10 with a margin of 10)."""
    mat = _matrix(cells, 2 * np.pi * 1e8 if cplx else 0.0)
    B = _rhs(mat.n, k)
    assert bool(_lib.lib().rb_femsolve_one_launch(mat.n, mat.struct.nnz, min(k, 128), int(cplx))) == one
    X, info = engine.solve(mat, B, coarse=False, groups=None)
    assert info["flag"] == 0 and (info["launches"] == 2) == one
    Y, info2 = engine.solve(mat, B, coarse=False)
    assert info2["flag"] == 0 and (info2["launches"] == 2) == one
    assert float((X - Y).abs().max()) <= 1e-10 * float(X.abs().max())
    if not cplx:
        Z, info3 = engine.solve(mat, B, coarse=False, groups=mat.mesh.row_groups())
        assert info3["flag"] == 0 and info3["launches"] > 2
        assert float((X - Z).abs().max()) <= 1e-10 * float(X.abs().max())


@pytest.mark.parametrize("omega", [0.0, 2 * np.pi * 1e8])
@pytest.mark.parametrize("start", [False, True])
def test_what_one_launch_does_not_solve_gets_the_coarse_space(omega, start):
    """21,112 nodes, 3 columns: one launch by default; capped at 10 iterations
    a sweep it stagnates, and the two-level form, which takes 80, answers."""
    mat = _matrix((28, 27, 25), omega)
    B = _rhs(mat.n, 3)
    want, info = engine.solve(mat, B)
    assert info["flag"] == 0 and info["launches"] == 2 and info["coarse_nc"] == 0
    x0 = 0.5 * want if start else None
    X, info = engine.solve(mat, B, maxiter=10, x0=x0)
    assert info["flag"] == 0 and info["coarse_nc"] > 0 and info["relres"] <= 1e-14
    assert float((X - want).abs().max()) <= 1e-10 * float(want.abs().max())
    assert engine.solve(mat, B, maxiter=10, coarse=False)[1]["flag"] == 1


def test_a_broken_dense_level_leaves_the_answer_to_jacobi():
    """A non-finite entry on a mesh below the coarse space's size: the cycle
    cannot set up its dense level, and the Jacobi solve reports the breakdown
    (flag 2) instead of an exception."""
    mat = _matrix((25, 25, 24))
    assert mat.n < engine.COARSE_MIN_NODES
    B = _rhs(mat.n, 64)
    assert engine.solve(mat, B)[1]["coarse_nc"] > 0  # the cycle's size
    at = int(mat.mesh.indptr[1000])
    mat.val64[at] = float("nan")
    mat.val32[at] = float("nan")
    _, info = engine.solve(mat, B)
    assert info["flag"] == 2 and info["coarse_nc"] == 0


@pytest.mark.parametrize("cells_max", [4096, 3])
def test_dense_level_of_a_batch_keeps_instances_apart(cells_max, monkeypatch):
    """However few aggregates are asked for, none holds rows of two instances;
    where the dense level cannot have that many, the batch solves by Jacobi."""
    from redbirdpy_b200.adjoint import BatchModel

    monkeypatch.setattr(engine, "mid_coarse_target", lambda ng: 1)
    cfgs = []
    for i in range(20):
        size = np.array([20, 18, 15]) * (1.0 + 0.1 * i)
        node, elem = kuhn_box(size, 1.0 + 0.1 * i)
        prop = np.tile([0.01, 1.0, 0.0, 1.37], (node.shape[0], 1))
        cfgs.append(rbb.meshprep(dict(node=node, elem=elem, prop=prop, srcpos=size[None] * [[0.4, 0.4, 0.0]],
                                      srcdir=np.array([[0, 0, 1.0]]), detpos=size[None] * [[0.6, 0.4, 0.0]],
                                      detdir=np.array([[0, 0, 1.0]]), omega=0.0))[0])
    bm = BatchModel(cfgs)
    monkeypatch.setattr(engine, "COARSE_MAX", cells_max)
    p = np.vstack([c["prop"] for c in cfgs])
    mua = torch.as_tensor(p[:, 0].copy(), device="cuda")
    mat = engine.assemble(bm.mesh, bm.optics(mua, 1.0 / (3.0 * (mua + 1.0))))
    mid = bm.mesh.mid_level()
    assert (mid is not None) == (cells_max > 3)
    if mid is not None:
        rows = mid.groups.rows[: 8 * mid.groups.ng].view(-1, 8).long()
        inst = bm.instances.row_inst.long()
        of_group = inst[rows[:, 0]]
        assert bool(((rows < 0) | (inst[rows.clamp_min(0)] == of_group[:, None])).all())
        agg = mid.coarse.agg[: mid.groups.ng].long()
        lo = torch.full((mid.coarse.nc,), 99, device="cuda").scatter_reduce(0, agg, of_group, "amin")
        hi = torch.full((mid.coarse.nc,), -1, device="cuda").scatter_reduce(0, agg, of_group, "amax")
        assert torch.equal(lo, hi)
    X, info = engine.solve(mat, bm.B, **bm.solve_kw)
    assert info["flag"] == 0 and not info["inst_status"].any() and (info["coarse_nc"] > 0) == (mid is not None)


def test_triangular_solves_that_finish_report_nothing():
    M = 700
    L = torch.eye(M, device="cuda", dtype=torch.float64)
    x = torch.ones(M, device="cuda", dtype=torch.float64)
    wb = _lib.lib().rb_chol_solve_work_bytes(M)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    engine.call("rb_chol_solve", engine.ptr(L), M, M, engine.ptr(x), engine.ptr(work), wb, engine.stream())
    engine.call("rb_chol_solve_status", engine.stream())
    assert bool((x == 1).all())


def test_one_launch_solves_build_no_row_groups(monkeypatch):
    """A default solve in one launch names its kernel and leaves the mesh's
    row groups unbuilt; a wide one builds and names them."""
    mat = _matrix((24, 22, 20))
    monkeypatch.setattr(engine.DeviceMesh, "mid_level", lambda self: None)
    _, info = engine.solve(mat, _rhs(mat.n, 4))
    assert info["product"] == info["spmm_kernel"] == "small_solve_kernel" and mat.mesh._groups is None
    _, info = engine.solve(mat, _rhs(mat.n, 128), coarse=False)
    assert info["product"] in ("spmm_blk_kernel", "small_solve_kernel")
    big = _matrix((32, 31, 30))
    _, info = engine.solve(big, _rhs(big.n, 128), coarse=False)
    assert info["product"] == "spmm_blk_kernel" and big.mesh._groups is not None


def test_plans_kept_on_a_mesh_are_finished_when_handed_out():
    """Another thread may use a kept plan on another stream at once: nothing
    of its making is under way on the stream that made it."""
    for build in ("row_groups", "mid_level", "coarse"):
        mesh = _matrix((60, 50, 40)).mesh
        torch.cuda.synchronize()
        plan = mesh.coarse_space(512) if build == "coarse" else getattr(mesh, build)()
        assert torch.cuda.current_stream().query() and plan is not None, build


def _slivers(m=(24, 24, 22)):
    """A Delaunay mesh with tets of 1e-6 of the cube, frequency domain."""
    from scipy.spatial import Delaunay

    rng = np.random.default_rng(0)
    g = np.stack(np.meshgrid(*[np.arange(float(k)) for k in m], indexing="ij"), -1).reshape(-1, 3)
    node = g + rng.uniform(-0.3, 0.3, g.shape)
    elem = Delaunay(node).simplices + 1
    x = node[elem - 1]
    vol = np.abs(np.einsum("ij,ij->i", np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), x[:, 3] - x[:, 0])) / 6
    node, elem = 2.0 * node, elem[vol > 1e-6]
    nn = node.shape[0]
    rng = np.random.default_rng(0)
    prop = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                            np.full(nn, 1.37)])
    pos = node.max(0)[None] * [[0.4, 0.4, 0.0]] + [[0, 0, 1e-3]]
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=pos, srcdir=np.array([[0, 0, 1.0]]), detpos=pos,
               detdir=np.array([[0, 0, 1.0]]), omega=2 * np.pi * 1e8)
    cfg, _ = rbb.meshprep(cfg)
    mesh = engine.mesh_of(cfg)
    return engine.assemble(mesh, engine.Optics.from_cfg(mesh, cfg))


def test_complex_columns_that_stall_in_one_launch_take_the_separate_kernels():
    """12,672 nodes x 16 on a mesh with slivers: the one-launch COCG stops at
    its cap and the separate kernels end the solve (flag 0, the reference FP64
    solve within the residual times a condition of 1e6); asked for one launch
    only, the outcome is what it is; a non-finite column is not retried."""
    mat = _slivers()
    B = _rhs(mat.n, 16)
    assert _lib.lib().rb_femsolve_one_launch(mat.n, mat.struct.nnz, 16, 1)
    X, info = engine.solve(mat, B)
    assert info["flag"] == 0 and info["launches"] > 2 and info["relres"] <= 1e-12
    Y, ref = engine.solve(mat, B, precision="fp64")
    assert ref["flag"] == 0
    assert float((X - Y).abs().max()) <= 1e-12 * 1e6 * float(Y.abs().max())
    easy = _matrix((20, 20, 20), 2 * np.pi * 1e8)
    C = _rhs(easy.n, 4)
    C[3, 1] = float("nan")
    _, info = engine.solve(easy, C)
    assert info["flag"] == 2 and info["launches"] == 2


def test_diverging_cycle_columns_end_their_sweep(monkeypatch):
    """COCG columns that diverge on a mesh with slivers are given up when
    their residual has grown to 1e8 of its start, long before the cap of 2000."""
    mat = _slivers((34, 32, 30))
    seen, real = [], engine.call

    def call(name, *a):
        real(name, *a)
        if name == "rb_femsolve_mid":
            seen.append((a[6]._obj.flag, a[6]._obj.sweep_iters_max, a[6]._obj.relres))

    monkeypatch.setattr(engine, "call", call)
    g = torch.Generator("cuda").manual_seed(128)
    B = torch.zeros((mat.n, 128), dtype=torch.float64, device="cuda")
    B.scatter_(0, torch.randint(0, mat.n, (4, 128), device="cuda", generator=g), 1.0)
    engine.solve(mat, B, maxiter=2000)
    assert len(seen) == 1
    flag, sweep, relres = seen[0]
    assert flag == 0 or (sweep < 1000 and relres < 1e9), seen
