"""The pipelined Jacobian kernel on long rows, also where the engine's rule
leaves such calls to the general kernel."""

import ctypes

import numpy as np
import pytest
import torch

import redbirdpy_b200 as rbb
from redbirdpy_b200 import _lib, engine

pytestmark = pytest.mark.gpu


def _delaunay_mesh():
    from scipy.spatial import Delaunay

    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(6.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    node = g + rng.uniform(-0.25, 0.25, g.shape)
    elem = Delaunay(node).simplices + 1
    x = node[elem - 1]
    vol = np.abs(np.einsum("ij,ij->i", np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), x[:, 3] - x[:, 0])) / 6
    cfg = dict(node=node, elem=elem[vol > 1e-6], prop=np.tile([0.01, 1.0, 0.0, 1.37], (node.shape[0], 1)),
               srcpos=np.array([[2.0, 2.0, 0]]), srcdir=np.array([[0, 0, 1.0]]), detpos=np.array([[3.0, 3.0, 0]]),
               detdir=np.array([[0, 0, 1.0]]), omega=0)
    return engine.mesh_of(rbb.meshprep(cfg)[0])


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ns,nd", [(3, 4), (4, 4), (12, 8), (5, 7), (28, 36), (40, 40), (64, 64)])
def test_pipelined_rows_equal_the_general_kernels(ns, nd, cplx):
    """Both quantities, bit for bit (same products, same order); sizes without
    a workspace (mostly empty tiles) run the general kernel either way."""
    mesh = _delaunay_mesh()
    assert 16 < mesh.rmax <= 32 and mesh.emax <= 64
    g = torch.Generator("cuda").manual_seed(7 * ns + nd)
    phi = torch.randn((mesh.nn, ns + nd), generator=g, device="cuda",
                      dtype=torch.complex128 if cplx else torch.float64)
    s, d = np.meshgrid(np.arange(ns), ns + np.arange(nd))
    cols, det0, ndet, psrc, pdet, colsd, ps, pd, _ = engine._pair_dev(
        np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)]), phi.device)
    whats = (_lib.RB_JAC_MUA_NODAL, _lib.RB_JAC_D)
    kind = _lib.RB_JAC_SPLIT_F32_ACC64 if cplx else _lib.RB_JAC_F32_ACC64
    ld = (2 * mesh.nn + 7) // 8 * 8
    out = []
    for wb in (_lib.lib().rb_jac_multi_work_bytes(mesh.rmax, ns, nd, int(cplx)), 0):
        J = torch.full(((2 if cplx else 1) * ns * nd, ld), float("nan"), device="cuda")
        work = torch.empty(max(wb, 16), dtype=torch.uint8, device="cuda")
        engine.call("rb_jac_multi", ctypes.byref(mesh.struct), 2, (ctypes.c_int32 * 2)(*whats),
                    (ctypes.c_int64 * 2)(0, mesh.nn), engine.ptr(phi), _lib.RB_C128 if cplx else _lib.RB_F64,
                    phi.shape[1], engine.ptr(colsd), len(cols), det0, ndet, engine.ptr(ps), engine.ptr(pd), -ns * nd,
                    engine.ptr(J), ld, kind, mesh.rmax, mesh.emax, engine.ptr(mesh.evol), engine.ptr(mesh.ddd), 0,
                    mesh.nn, engine.ptr(work) if wb else None, wb, engine.stream())
        engine._jac_checked()
        out.append(J[:, :2 * mesh.nn])
    assert torch.equal(out[0], out[1])
