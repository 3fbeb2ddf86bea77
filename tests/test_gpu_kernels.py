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
