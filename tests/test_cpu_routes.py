"""Host-side choice of routes, with the library's calls recorded."""

import types

import numpy as np
import pytest
import torch

from redbirdpy_b200 import engine


def _jac_calls(monkeypatch, nn, ns, nd, cplx, params, acc64=True, grid=True):
    """(names of the library calls, their pair counts, J) of one jacobian_matrix call."""
    log = []
    monkeypatch.setattr(engine, "call", lambda name, *a: log.append((name, a)))
    monkeypatch.setattr(engine, "stream", lambda: None)
    monkeypatch.setattr(engine, "_jac_checked", lambda: None)
    mesh = types.SimpleNamespace(nn=nn, struct=engine._lib.RbMesh(), rmax=15, emax=24, evol=None, ddd=None)
    s, d = np.meshgrid(np.arange(ns), ns + np.arange(nd))
    sd = np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)])
    if not grid:
        sd = sd[:-1]
    phi = torch.zeros((nn, ns + nd), dtype=torch.complex128 if cplx else torch.float64)
    J, K = engine.jacobian_matrix(mesh, phi, sd, params, "exact", acc64=acc64)
    assert K == len(params) * nn
    counts = [a[11] if name == "rb_jac_range" else a[13] for name, a in log]
    return [name for name, _ in log], counts, J


@pytest.mark.parametrize("cplx", [False, True])
def test_jacobian_rows_below_the_line_take_the_general_kernel_alone(cplx, monkeypatch):
    """Small meshes, other pair tables and other row types: rb_jac's own
    preparation and row stride, nothing of the pipelined kernel's."""
    asked = []
    real = engine._grid_nsd
    monkeypatch.setattr(engine, "_grid_nsd", lambda *a: asked.append(a[4:]) or real(*a))
    w = 2 if cplx else 1
    names, counts, J = _jac_calls(monkeypatch, 2002, 5, 7, cplx, ("mua", "D"))
    assert names == ["rb_jac_range"] * 2 and counts == [35, 35] and asked == [()]
    assert J.stride(0) == 4004 and J.shape[0] == 35 * w
    names, counts, J = _jac_calls(monkeypatch, 2002, 4, 8, cplx, ("mua",))
    assert names == ["rb_jac_range"] and counts == [-32] and J.stride(0) == 2004
    names, counts, J = _jac_calls(monkeypatch, 9001, 16, 16, cplx, ("mua",), acc64=False)
    assert names == ["rb_jac_range"] and counts == [-256] and J.stride(0) == 9004
    names, counts, J = _jac_calls(monkeypatch, 9001, 16, 16, cplx, ("mua",), grid=False)
    assert names == ["rb_jac_range"] and counts == [255] and J.stride(0) == 9004
    assert _jac_calls(monkeypatch, 9001, 16, 16, cplx, ())[0] == []


@pytest.mark.parametrize("cplx", [False, True])
def test_jacobian_rows_of_the_full_grid_take_the_pipelined_kernel(cplx, monkeypatch):
    names, counts, J = _jac_calls(monkeypatch, 9001, 15, 16, cplx, ("mua", "D"))
    assert names == ["rb_jac_multi"] and counts == [-240] and J.stride(0) == 18008


@pytest.mark.parametrize("refine,norms,checked", [(0, [], True), (3, [1.0, 1e-3, 1e-15], False),
                                                  (3, [1.0, 1e-3, 1e-6, 1e-9], True), (2, [1.0, float("nan"), 1.0], True)])
def test_normal_solve_asks_after_waits_that_gave_up(refine, norms, checked, monkeypatch):
    """A triangular solve whose result no finite residual vouches for is asked
    whether a wait gave up; its error reaches the caller."""
    log, fail = [], []

    def call(name, *a):
        log.append(name)
        if name == "rb_chol_solve_status" and fail:
            raise engine._lib.RedbirdError(name, engine._lib.RB_ECUDA, "a wait gave up")

    class Op(engine.StoredJacobian):
        def __init__(self, J, K, lo):
            self.rows = J.shape[0]

        def jt_then_j(self, y):
            return torch.zeros(9), torch.zeros(self.rows)

        def jt(self, y, alpha):
            return torch.zeros(9)

    monkeypatch.setattr(engine, "call", call)
    monkeypatch.setattr(engine, "stream", lambda: None)
    monkeypatch.setattr(engine, "StoredJacobian", Op)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    H, di, r = torch.zeros((4, 4), dtype=torch.float64), torch.ones(4, dtype=torch.float64), np.ones(4)
    for broken in (False, True):
        log.clear()
        fail[:] = [1] * broken
        left = list(norms)
        monkeypatch.setattr(engine, "norm2", lambda t: left.pop(0))
        if broken and checked:
            with pytest.raises(engine._lib.RedbirdError):
                engine.normal_solve(torch.zeros((4, 9)), 9, H, di, r, 0.1, refine=refine)
        else:
            engine.normal_solve(torch.zeros((4, 9)), 9, H, di, r, 0.1, refine=refine)
        assert log.count("rb_chol_solve_status") == checked


@pytest.mark.parametrize("rmax,emax,ns,nd,cplx,wins", [
    (15, 24, 3, 4, False, 0), (15, 24, 4, 4, False, 1), (15, 24, 3, 4, True, 1), (15, 24, 64, 64, True, 1),
    (25, 44, 4, 4, False, 0), (25, 44, 12, 12, False, 0), (25, 44, 12, 16, False, 1), (24, 42, 5, 7, True, 0),
    (25, 44, 16, 16, True, 1), (25, 44, 64, 64, True, 1), (25, 44, 61, 64, False, 1), (25, 44, 40, 40, False, 0),
    (25, 44, 64, 48, False, 1), (25, 44, 64, 64, False, 0), (29, 44, 64, 64, False, 1), (40, 44, 64, 64, True, 0),
    (25, 70, 64, 64, True, 0)])
def test_rows_of_long_neighbour_lists_take_the_faster_kernel(rmax, emax, ns, nd, cplx, wins):
    """The line between the general and the pipelined Jacobian kernel on
    meshes off the box (17 to 32 neighbours), on both sides of each of its terms."""
    assert engine._lib.lib().rb_jac_multi_wins(rmax, emax, ns, nd, int(cplx)) == wins


@pytest.mark.parametrize("k,cplx,form,name", [
    (7, False, "cycle", "spmm_kernel"), (65, False, "cycle", "vc_spmm_kernel"), (125, True, "cycle", "spmm_pair_kernel"),
    (64, True, "cycle", "spmm_kernel"), (3, True, "one", "small_solve_kernel"), (67, False, "groups", "spmm_blk_kernel"),
    (64, False, "groups", "spmm_kernel"), (66, False, "rows", "spmm_pair_kernel"), (128, True, "rows", "spmm_pair_kernel"),
    (100, True, "rows", "spmm_kernel")])
def test_product_names_follow_the_dispatch(k, cplx, form, name):
    assert engine._product_kernel(40000, k, cplx, engine._lib.RB_MIXED, form) == name


def test_fp64_product_names():
    assert engine._product_kernel(9, 64, False, engine._lib.RB_FP64, "rows") == "spmm_grp_kernel"
    assert engine._product_kernel(9, 63, False, engine._lib.RB_FP64, "rows") == "spmm_grp_kernel"
    assert engine._product_kernel(9, 48, False, engine._lib.RB_FP64, "rows") == "spmm_kernel"
