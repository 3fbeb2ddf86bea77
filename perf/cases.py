"""What a program built on this package asks of it, as cases that can be timed and checked.

Six kinds of work, each through a public entry point: the forward model
(``runforward`` from host arrays, ``forward_device`` on the GPU), the adjoint
gradient of one model and of a batch of uneven ones (``detector_values`` and
its backward), the Gauss-Newton Jacobian rows (``jacobian_matrix``), the
regularised normal equations (``row_sumsq`` and ``reginv_under_device``) and a
whole reconstruction iteration (``runrecon``).  Meshes are boxes of Kuhn
tetrahedra, the repository's own workloads, with regular or displaced nodes;
``exact`` restates each result in FP64 with plain torch.
"""

import functools
import math

import numpy as np
import torch

import redbirdpy_b200 as rb
from redbirdpy_b200 import engine
from redbirdpy_b200.adjoint import BatchModel, DeviceModel, detector_values
from redbirdpy_b200.forward import forward_device
from redbirdpy_b200.meshgen import batch_boxes, grid_optodes, kuhn_box

C0 = 299792458000.0  # mm/s
OMEGA = 2 * math.pi * 1e8  # 100 MHz modulation of the frequency-domain cases
REFF, NREF = 0.493, 1.37
BULK = {"mua": 0.01, "musp": 1.0, "n": NREF}


def _mesh(nx, ny, nz, h, jitter=False):
    return {"nx": nx, "ny": ny, "nz": nz, "h": h, "jitter": jitter}


def listed():
    return [
        # a first simulation at the keyboard: 1,183 nodes, one source, two detectors; launches and host calls
        dict(name="forward_tiny", op="forward", host=True, prop="label", fd=False, ns=1, nd=2, **_mesh(12, 12, 6, 5.0)),
        # one small probe in the frequency domain, odd counts, properties per node, unstructured node positions
        dict(name="forward_small_fd", op="forward", host=True, prop="node", fd=True, ns=5, nd=7,
             **_mesh(20, 16, 10, 2.0, True)),
        # an ordinary subject mesh (43k nodes) with a number of columns that fits no lane layout
        dict(name="forward_ragged", op="forward", host=True, prop="node", fd=False, ns=17, nd=20,
             **_mesh(48, 41, 20, 2.0, True)),
        # the large imaging array: 3M tets, 64 sources and 64 detectors, continuous wave
        dict(name="forward_large", op="forward", host=False, prop="label", fd=False, ns=64, nd=64,
             **_mesh(100, 100, 50, 1.0)),
        # the same array in the frequency domain
        dict(name="forward_large_fd", op="forward", host=False, prop="node", fd=True, ns=64, nd=64,
             **_mesh(100, 100, 50, 1.0)),
        # one step of a gradient-based fit: 375k tets, 32 x 32 pairs
        dict(name="gradient", op="gradient", fd=False, ns=32, nd=32, **_mesh(50, 50, 25, 2.0)),
        # the same on a smaller frequency-domain model with odd counts
        dict(name="gradient_fd_odd", op="gradient", fd=True, ns=13, nd=9, **_mesh(30, 26, 14, 2.0, True)),
        # a training batch: 64 uneven models in one block-diagonal system
        dict(name="gradient_batch", op="batch", count=64, boxes=2),
        # Jacobian rows of a 64 x 64 frequency-domain array for mua and D: 8192 rows, 135,252 columns
        dict(name="jacobian_fd", op="jacobian", fd=True, ns=64, nd=64, **_mesh(50, 50, 25, 2.0)),
        # the regularised normal equations of such rows
        dict(name="normal_equations", op="normal", rows=8192, cols=135252),
        # one reconstruction iteration on a small probe, absorption alone, odd counts
        dict(name="recon_small", op="recon", fd=False, param="mua", ns=11, nd=13, **_mesh(30, 25, 13, 2.0, True)),
        # one reconstruction iteration of the large array: 8192 rows, 1,040,502 unknowns
        dict(name="recon_large", op="recon", fd=True, param="mua+D", ns=64, nd=64, **_mesh(100, 100, 50, 1.0)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, lo, hi):
    """A box of about lo..hi nodes (over the logarithm), uneven extents."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.8, 1.25), rng.uniform(0.4, 0.8)
    e = (n / (a * b)) ** (1 / 3)
    nx, ny, nz = (max(4, int(round(e * f)) - 1) for f in (1.0, a, b))
    h = round(min(5.0, 90.0 / nx), 3)
    return _mesh(nx, ny, nz, h, rng.random() < 0.5)


def draw(rng):
    op = rng.choice(["forward", "forward", "forward", "gradient", "batch", "jacobian", "normal", "recon"])
    fd = rng.random() < 0.5
    if op == "forward":
        host = rng.random() < 0.5
        return dict(op=op, host=host, prop=rng.choice(["label", "node"]), fd=fd, ns=_log_int(rng, 1, 64),
                    nd=_log_int(rng, 1, 64), **_draw_mesh(rng, 1200, 60000 if host else 500000))
    if op == "gradient":
        return dict(op=op, fd=fd, ns=_log_int(rng, 2, 32), nd=_log_int(rng, 2, 32), **_draw_mesh(rng, 2000, 70000))
    if op == "batch":
        return dict(op=op, count=_log_int(rng, 4, 64), boxes=rng.randrange(1000))
    if op == "jacobian":
        return dict(op=op, fd=fd, ns=_log_int(rng, 4, 64), nd=_log_int(rng, 4, 64), **_draw_mesh(rng, 2000, 60000))
    if op == "normal":
        rows = _log_int(rng, 64, 8192)
        return dict(op=op, rows=rows, cols=_log_int(rng, max(2000, rows + 1), 135000))
    return dict(op=op, fd=fd, param=rng.choice(["mua", "mua+D"]), ns=_log_int(rng, 3, 16), nd=_log_int(rng, 3, 16),
                **_draw_mesh(rng, 4000, 40000))


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=2)
def _box(nx, ny, nz, h):
    return kuhn_box(np.array([nx, ny, nz]) * h, h)


def _cfg(case, rng):
    """An unprepared cfg dict: mesh, optodes on the top face, properties."""
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["h"]
    node, elem = _box(nx, ny, nz, h)
    node, elem = node.copy(), elem.copy()
    size = np.array([nx, ny, nz]) * h
    if case["jitter"]:  # interior nodes off the grid, as a mesh generator leaves them
        inside = np.all((node > 0.5 * h) & (node < size - 0.5 * h), axis=1)
        node[inside] += rng.uniform(-0.12, 0.12, (int(inside.sum()), 3)) * h

    def optodes(k, shift):
        side = math.ceil(math.sqrt(k))
        p = grid_optodes([0.15 * size[0], 0.85 * size[0]], [0.15 * size[1], 0.85 * size[1]], side)[:k]
        p[:, :2] += shift + rng.uniform(-0.3, 0.3, (k, 2)) * h
        return p

    cfg = dict(node=node, elem=elem, srcpos=optodes(case["ns"], 0.0), srcdir=np.array([[0, 0, 1.0]]),
               detpos=optodes(case["nd"], 0.05 * size[0]), detdir=np.array([[0, 0, 1.0]]),
               omega=OMEGA if case["fd"] else 0.0, reff=REFF, bulk=BULK)
    if case.get("prop") == "label":
        cfg["prop"] = np.array([[0, 0, 1, 1], [rng.uniform(0.008, 0.012), rng.uniform(0.9, 1.1), 0, NREF]])
        cfg["seg"] = np.ones(elem.shape[0], dtype=np.int32)
    elif case["op"] == "recon":  # homogeneous starting point of a reconstruction
        cfg["prop"] = np.tile([0.01, 1.0, 0.0, NREF], (node.shape[0], 1))
    else:
        nn = node.shape[0]
        cfg["prop"] = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                                       np.full(nn, NREF)])
    return cfg


def _truth(case, node, rng):
    """The properties behind the measured data: two spherical inclusions."""
    size = np.array([case["nx"], case["ny"], case["nz"]]) * case["h"]
    prop = np.tile([0.01, 1.0, 0.0, NREF], (node.shape[0], 1))
    r = 0.16 * size.min() * rng.uniform(0.9, 1.1)
    prop[np.linalg.norm(node - size * [0.35, 0.5, 0.4], axis=1) < r, 0] = 0.025
    prop[np.linalg.norm(node - size * [0.65, 0.5, 0.5], axis=1) < r, 1] = 2.0
    return prop


def _noise(shape, fd, rng):
    """1% amplitude noise and, in the frequency domain, 0.5 degree of phase."""
    n = 1 + 0.01 * rng.standard_normal(shape)
    return n * np.exp(1j * np.deg2rad(0.5) * rng.standard_normal(shape)) if fd else n


def _batch_cfgs(case, seed):
    """The case's boxes and optodes with properties of the seed's own."""
    rng = np.random.default_rng(seed)
    cfgs = [dict(c, reff=REFF, bulk=BULK) for c in batch_boxes(case["count"], case["boxes"])]
    for c in cfgs:
        nn = c["node"].shape[0]
        c["prop"] = np.column_stack([rng.uniform(0.005, 0.03, nn), rng.uniform(0.5, 2.0, nn), np.zeros(nn),
                                     np.full(nn, NREF)])
    return cfgs


def _optical(cfgs):
    p = np.vstack([np.atleast_2d(c["prop"]) for c in cfgs])
    return (torch.as_tensor(p[:, 0].copy(), device="cuda"),
            torch.as_tensor(1.0 / (3.0 * (p[:, 0] + p[:, 1])), device="cuda"))


def _near(cfgs):
    """The pairs a fit uses: detector rows of every model against source
    columns, its own pairs within 40 mm (beyond, a measurement is noise)."""
    ns = max(len(c["srcpos"]) for c in cfgs)
    rows = [np.linalg.norm(np.asarray(c["detpos"])[:, None] - np.asarray(c["srcpos"])[None], axis=2) < 40.0
            for c in cfgs]
    return torch.as_tensor(np.vstack([np.pad(r, ((0, 0), (0, ns - r.shape[1]))) for r in rows]), device="cuda")


def _medium_fields(node, pts, fd):
    """nn x npts fields of point optodes in an infinite medium, FP64."""
    mua, d = 0.01, 1.0 / 3.03
    k = np.sqrt(complex(mua, OMEGA * NREF / C0 if fd else 0.0) / d)
    r = torch.cdist(torch.as_tensor(node, device="cuda"), torch.as_tensor(pts, device="cuda"),
                    compute_mode="donot_use_mm_for_euclid_dist").clamp_min(0.5)
    amp = torch.exp(-k.real * r) / (4 * math.pi * d * r)
    return torch.polar(amp, -k.imag * r) if fd else amp


def _moved(pos):
    """Optodes one transport length below the surface, as the package places them."""
    return pos + np.array([0, 0, 1.0 / 1.01])


def _pairs(ns, nd):
    """The source-detector table, detector-major, all pairs active."""
    s, d = np.meshgrid(np.arange(ns), ns + np.arange(nd))
    return np.column_stack([s.ravel(), d.ravel(), np.ones(ns * nd)])


def _normal_inputs(case, seed):
    """(J, r): FP32 rows with the decay of measured sensitivities, the row
    stride padded to 16 bytes, and the misfit of a small inclusion."""
    g = torch.Generator("cuda").manual_seed(seed)
    M, K = case["rows"], case["cols"]
    ns = max(1, int(math.isqrt(M)))
    box = torch.tensor([100.0, 100.0, 50.0], device="cuda")
    pos = torch.rand((K, 3), generator=g, device="cuda") * box
    opt = torch.rand((2 * ns + 2, 3), generator=g, device="cuda") * box * torch.tensor([1.0, 1.0, 0.0], device="cuda")
    r = torch.cdist(opt, pos, compute_mode="donot_use_mm_for_euclid_dist").clamp_min(1.0)
    f = torch.exp(-0.17 * r) / r
    sign = torch.cos(0.05 * r)
    ld = (K + 3) // 4 * 4
    J = torch.zeros((M, ld), dtype=torch.float32, device="cuda")
    for a in range(0, M, 512):
        k = torch.arange(a, min(M, a + 512), device="cuda")
        s, d = k % (ns + 1), ns + 1 + (k // (ns + 1)) % (ns + 1)
        J[k, :K] = -f[s] * f[d] * torch.where((k < M // 2)[:, None], sign[s] * sign[d], sign[s] - 0.9 * sign[d])
    x = 0.01 * torch.exp(-((pos - box / 2) ** 2).sum(1) / 100).double()
    y = torch.cat([J[a:a + 512, :K].double() @ x for a in range(0, M, 512)])
    y = y * (1 + 0.01 * torch.randn(M, generator=g, device="cuda", dtype=torch.float64))
    return J, y.cpu().numpy()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    op = case["op"]
    if op == "normal":
        J, r = _normal_inputs(case, seed)
        return {"case": case, "J": J, "r": r}
    if op == "batch":
        cfgs = [rb.meshprep(c)[0] for c in _batch_cfgs(case, seed)]
        model = BatchModel(cfgs)
        mua, dco = _optical(cfgs)
        with torch.no_grad():
            target = detector_values(model, mua * 1.1, dco)
        return {"case": case, "model": model, "mua": mua, "D": dco, "target": target, "own": _near(cfgs)}
    cfg, sd = rb.meshprep(_cfg(case, rng))
    if op == "gradient":
        model = DeviceModel(cfg)
        mua, dco = _optical([cfg])
        with torch.no_grad():
            target = detector_values(model, mua * 1.1, dco)
        return {"case": case, "model": model, "mua": mua, "D": dco, "target": target, "own": _near([cfg])}
    if op == "jacobian":
        phi = _medium_fields(cfg["node"], _moved(np.vstack([cfg["srcpos"], cfg["detpos"]])), case["fd"])
        mesh = engine.mesh_of(cfg)
        mesh.ddd, mesh.evol  # the geometry of a mesh in use
        return {"case": case, "mesh": mesh, "phi": phi, "sd": sd}
    if op == "recon":
        truth = dict(cfg, prop=_truth(case, cfg["node"], rng))
        data = forward_device(truth)[0].cpu().numpy()
        return {"case": case, "cfg": cfg, "sd": sd, "data": data * _noise(data.shape, case["fd"], rng)}
    return {"case": case, "cfg": cfg}


def _loss(det, target, own):
    """Log-amplitude misfit over the pairs of ``own``."""
    one = torch.ones_like(det)
    d, t = torch.where(own, det, one), torch.where(own, target, one)
    return 0.5 * torch.sum((torch.log(torch.abs(d)) - torch.log(torch.abs(t))) ** 2)


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "forward":
        if case["host"]:
            det, phi = rb.runforward(state["cfg"])
        else:
            det, phi = forward_device(state["cfg"])[:2]
        return {"det": det, "phi": phi}
    if op in ("gradient", "batch"):
        mua, dco = state["mua"].clone().requires_grad_(True), state["D"].clone().requires_grad_(True)
        det = detector_values(state["model"], mua, dco)
        _loss(det, state["target"], state["own"]).backward()
        return {"det": torch.where(state["own"], det.detach(), torch.zeros_like(det)), "mua": mua.grad, "D": dco.grad}
    if op == "jacobian":
        J, K = engine.jacobian_matrix(state["mesh"], state["phi"], state["sd"], ("mua", "D"), "exact", acc64=True)
        return J[:, :K]
    if op == "normal":
        J, K = state["J"], case["cols"]
        rowsq, total, Jb = engine.row_sumsq(J, K, bf16_copy=True)
        return engine.reginv_under_device(J, K, state["r"], 0.0, 1.0 / float(total.item()), "bf16", lam_rel=0.05,
                                          rowsq=rowsq, Jb=Jb)
    cfg = dict(state["cfg"])
    recon, resid, _, updates, J, det, phi = rb.runrecon(
        cfg, {"prop": cfg["prop"].copy()}, state["data"], state["sd"], maxiter=1, report=False, param=case["param"],
        lambda_rule="maxdiag")
    out = {"resid": resid, "prop": recon["prop"], "update": updates[0], "det": det, "phi": phi}
    if not torch.is_tensor(J["mua"]):  # rows handed to the host; the largest stay where they are
        out["J"] = J["mua"]
    return out


# --------------------------------------------------------------------- work
def _mesh_counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nn, ne = (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz
    return nn, ne


def _forward_work(nn, ne, k, w):
    """Mesh (nodes, tets, properties) in, fields out; one product with the
    matrix's ~15 entries per row is the least that touches every column."""
    return {"bytes": 16 * ne + 48 * nn + w * nn * k, "flops": (2 if w == 8 else 8) * 15 * nn * k}


def work(case):
    op = case["op"]
    if op == "batch":
        n = 10600 * case["count"]  # mean nodes of an instance over the drawn extents and spacings
        f = _forward_work(n, 5.3 * n, 32, 8)
        return {"bytes": f["bytes"] + 32 * n, "flops": 2 * f["flops"]}
    if op == "normal":
        M, K = case["rows"], case["cols"]
        return {"bytes": 4 * M * K + 8 * K + 8 * M, "flops": M * M * K + M ** 3 / 3 + 4 * M * K}
    nn, ne = _mesh_counts(case)
    fd, ns, nd = case["fd"], case["ns"], case["nd"]
    f = _forward_work(nn, ne, ns + nd, 16 if fd else 8)
    if op == "forward":
        return f
    if op == "gradient":
        return {"bytes": f["bytes"] + 32 * nn, "flops": f["flops"] + (8 if fd else 2) * 30 * nn * ns}
    rows = ns * nd * (2 if fd else 1)
    cols = nn if op == "recon" and case["param"] == "mua" else 2 * nn
    j = {"bytes": 4 * rows * cols, "flops": (8 if fd else 2) * 15 * cols * ns * nd}
    if op == "jacobian":
        return {"bytes": j["bytes"] + 16 * ne + f["bytes"], "flops": j["flops"]}
    return {"bytes": f["bytes"] + 16 * cols, "flops": f["flops"] + j["flops"] + rows * rows * cols + rows ** 3 / 3}


# -------------------------------------------------------------------- exact
class _Fem:
    """The P1 diffusion model on one mesh in plain FP64 torch."""

    def __init__(self, node, elem, fd):
        self.x = torch.as_tensor(node, device="cuda")
        self.e = torch.as_tensor(elem[:, :4].astype(np.int64) - 1, device="cuda")
        self.nn, self.ne, self.fd = self.x.shape[0], self.e.shape[0], fd
        p = self.x[self.e]
        self.edges = (p[:, 1:] - p[:, :1]).transpose(1, 2)  # columns x_i - x_0
        inv = torch.linalg.inv(self.edges)
        self.inv = inv
        self.vol = torch.linalg.det(self.edges).abs() / 6
        grad = torch.cat([-inv.sum(1, keepdim=True), inv], 1)
        self.ddd = torch.einsum("eik,ejk->eij", grad, grad) * self.vol[:, None, None]
        f = torch.cat([self.e[:, [0, 1, 2]], self.e[:, [0, 1, 3]], self.e[:, [0, 2, 3]], self.e[:, [1, 2, 3]]])
        f = f.sort(1).values
        key, cnt = torch.unique((f[:, 0] * self.nn + f[:, 1]) * self.nn + f[:, 2], return_counts=True)
        key = key[cnt == 1]
        self.f = torch.stack([key // self.nn // self.nn, key // self.nn % self.nn, key % self.nn], 1)
        q = self.x[self.f]
        self.area = 0.5 * torch.linalg.norm(torch.linalg.cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0]), dim=1)

    def matrix(self, mua, d, per_node=True):
        """CSR matrix for nodal (or, per_node False, uniform) mua and D."""
        two = 1 + torch.eye(4, dtype=torch.float64, device="cuda")
        v = self.vol[:, None, None]
        if per_node:
            m, de = mua[self.e], d[self.e].mean(1)
            w = (m.sum(1)[:, None, None] + m[:, :, None] + m[:, None, :]) / 120 * two * v
        else:
            de, w = d, 0.05 * mua * two * v
        a = self.ddd * (de[:, None, None] if per_node else de) + w
        if self.fd:
            a = a + 1j * (OMEGA / C0 * NREF * 0.05) * two * v
        b = (self.area * (1 - REFF) / (12 * (1 + REFF)))[:, None, None] * 0.5 * two[:3, :3]
        i = torch.cat([self.e[:, :, None].expand(-1, 4, 4).reshape(-1), self.f[:, :, None].expand(-1, 3, 3).reshape(-1)])
        j = torch.cat([self.e[:, None, :].expand(-1, 4, 4).reshape(-1), self.f[:, None, :].expand(-1, 3, 3).reshape(-1)])
        val = torch.cat([a.reshape(-1), b.reshape(-1).to(a.dtype)])
        return torch.sparse_coo_tensor(torch.stack([i, j]), val, (self.nn, self.nn)).coalesce().to_sparse_csr()

    def weights(self, pts, lo=0, hi=None):
        """nn x npts barycentric weights of points among tets lo..hi-1."""
        out = torch.zeros((self.nn, len(pts)), dtype=torch.float64, device="cuda")
        for k, p in enumerate(torch.as_tensor(pts, device="cuda")):
            l3 = torch.einsum("eij,ej->ei", self.inv[lo:hi], p - self.x[self.e[lo:hi, 0]])
            b = torch.cat([1 - l3.sum(1, keepdim=True), l3], 1)
            t = int(b.min(1).values.argmax())
            out[self.e[lo + t], k] = b[t]
        return out

    def solve(self, A, B):
        """A X = B: dense for small systems, else refined Jacobi CG / COCG."""
        B = B.to(torch.complex128 if self.fd else torch.float64)
        if self.nn <= 6000:
            return torch.linalg.solve(A.to_dense(), B)
        ip, ix, va = A.crow_indices(), A.col_indices(), A.values()
        row = torch.repeat_interleave(torch.arange(self.nn, device="cuda"), ip[1:] - ip[:-1])
        dinv = (1 / va[row == ix])[:, None]

        def quot(a, b):
            return torch.where(b != 0, a / torch.where(b != 0, b, torch.ones_like(b)), torch.zeros_like(a))

        X = torch.zeros_like(B)
        for _ in range(4):
            r = B - A @ X
            x, p, rz = torch.zeros_like(r), None, None
            stop = 1e-5 * torch.linalg.norm(r, dim=0)
            for it in range(600):
                if it % 10 == 0 and bool((torch.linalg.norm(r, dim=0) <= stop).all()):
                    break
                z = dinv * r
                new = (r * z).sum(0)
                p = z if p is None else z.addcmul_(p, quot(new, rz)[None])
                rz = new
                q = A @ p
                al = quot(rz, (p * q).sum(0))[None]
                x.addcmul_(p, al)
                r.addcmul_(q, -al)
            X += x
        return X

    def pair_terms(self, s, d, reference=False):
        """Sensitivities of phi_s^T (-dA) phi_d by node: yields (nodes, mua
        terms, D terms) for a chunk of tets, the pairs (s, d) of s: nn x S and
        d: nn x D in the last axes (detector, source)."""
        S, D = s.shape[1], d.shape[1]
        chunk = max(1, (1 << 27) // (S * D))
        for a in range(0, self.ne, chunk):
            e, v = self.e[a:a + chunk], self.vol[a:a + chunk, None, None]
            fs, fd = s[e], d[e]  # tets x 4 x columns
            ts, td = fs.sum(1), fd.sum(1)
            same = torch.einsum("eid,eis->eds", fd, fs)
            both = td[:, :, None] * ts[:, None, :] + same
            gd = torch.einsum("eij,eid->ejd", self.ddd[a:a + chunk].to(fd.dtype), fd)
            dd = -0.25 * torch.einsum("ejd,ejs->eds", gd, fs)
            for n in range(4):
                if reference:
                    m = -0.0125 * v * both
                else:
                    m = -v / 120 * (both + fd[:, n, :, None] * (ts + fs[:, n])[:, None, :]
                                    + (td + fd[:, n])[:, :, None] * fs[:, n, None, :])
                yield e[:, n], m, dd

    def jacobian(self, s, d, reference=False):
        """(Jmua, JD) rows x nodes, pairs detector-major."""
        n = s.shape[1] * d.shape[1]
        out = [torch.zeros((self.nn, n), dtype=s.dtype, device="cuda") for _ in range(1 if reference else 2)]
        for nodes, *terms in self.pair_terms(s, d, reference):
            for o, t in zip(out, terms):
                o, t = (torch.view_as_real(o), torch.view_as_real(t)) if t.is_complex() else (o, t)
                o.index_add_(0, nodes, t.reshape(t.shape[0], *o.shape[1:]))
        return [o.T for o in out]

    def gradient(self, s, lam):
        """sum over columns of the nodal sensitivities of the pairs (s_j, lam_j)."""
        out = torch.zeros((2, self.nn), dtype=torch.float64, device="cuda")
        for j in range(s.shape[1]):
            for nodes, m, dd in self.pair_terms(s[:, j:j + 1], lam[:, j:j + 1]):
                out[0].index_add_(0, nodes, m.real.reshape(-1))
                out[1].index_add_(0, nodes, dd.real.reshape(-1))
        return out


def _exact_gradient(fem, Bs, Bd, mua, dco, own):
    """own: the nd x ns pairs (detector rows, source columns) of the loss."""

    def fields(m):
        X = fem.solve(fem.matrix(m, dco), torch.cat([Bs, Bd], 1))
        ph, pd = X[:, :Bs.shape[1]], X[:, Bs.shape[1]:]
        return ph, pd, Bd.to(ph.dtype).T @ ph
    target = fields(mua * 1.1)[2]
    ph, pd, det = fields(mua)
    leaf = det.clone().requires_grad_(True)
    _loss(leaf, target, own).backward()
    lam = pd @ leaf.grad.conj()
    g = fem.gradient(ph, lam)
    return {"det": torch.where(own, det, torch.zeros_like(det)), "mua": g[0], "D": g[1]}


def _exact_batch(case, seed):
    cfgs = _batch_cfgs(case, seed)
    off = np.cumsum([0] + [c["node"].shape[0] for c in cfgs])
    fem = _Fem(np.vstack([c["node"] for c in cfgs]), np.vstack([c["elem"] + o for c, o in zip(cfgs, off)]), False)
    S, nd = max(len(c["srcpos"]) for c in cfgs), [len(c["detpos"]) for c in cfgs]
    Dm, D0 = max(nd), np.cumsum([0] + nd)
    Bs = torch.zeros((fem.nn, S), dtype=torch.float64, device="cuda")
    Bd = torch.zeros((fem.nn, Dm), dtype=torch.float64, device="cuda")
    own, lo = _near(cfgs), 0
    for i, c in enumerate(cfgs):
        hi = lo + c["elem"].shape[0]
        Bs[:, :len(c["srcpos"])] += fem.weights(_moved(c["srcpos"]), lo, hi)
        Bd[:, :nd[i]] += fem.weights(_moved(c["detpos"]), lo, hi)
        lo = hi
    mua, dco = _optical(cfgs)

    def rows(f):  # per instance: its detector columns against every source column
        return torch.cat([Bd[a:b, :k].T @ f[a:b] for a, b, k in zip(off[:-1], off[1:], nd)])

    def fields(m):
        X = fem.solve(fem.matrix(m, dco), torch.cat([Bs, Bd], 1))
        return X[:, :S], X[:, S:], rows(X[:, :S])
    target = fields(mua * 1.1)[2]
    ph, pd, det = fields(mua)
    leaf = det.clone().requires_grad_(True)
    _loss(leaf, target, own).backward()
    lam = torch.cat([pd[a:b, :k] @ leaf.grad[r:r + k] for a, b, k, r in zip(off[:-1], off[1:], nd, D0)])
    g = fem.gradient(ph, lam)
    return {"det": torch.where(own, det, torch.zeros_like(det)), "mua": g[0], "D": g[1]}


def _regularised(J, r, lam_rel):
    """alpha J^T (alpha J J^T + lam I)^-1 r, alpha = 1 / ||J||_F^2, lam = lam_rel max diag."""
    al = 1 / sum(float(b.double().square().sum()) for b in J.split(512))
    H = torch.zeros((J.shape[0],) * 2, dtype=torch.float64, device="cuda")
    for c in J.split(8192, dim=1):
        c = c.double()
        H.addmm_(c, c.T, alpha=al)
    H.diagonal().add_(lam_rel * float(H.diagonal().max()))
    y = torch.cholesky_solve(r[:, None], torch.linalg.cholesky(H))
    return al * torch.cat([c.double().T @ y[:, 0] for c in J.split(8192, dim=1)])


def exact(case, seed):
    op = case["op"]
    if op == "normal":
        J, r = _normal_inputs(case, seed)
        return _regularised(J[:, :case["cols"]], torch.as_tensor(r, device="cuda"), 0.05)
    if op == "batch":
        return _exact_batch(case, seed)
    if op == "recon" and _mesh_counts(case)[0] > 100000:
        return None  # an FP64 Gauss-Newton step of this size takes minutes in plain torch
    rng = np.random.default_rng(seed)
    cfg = _cfg(case, rng)
    fem = _Fem(cfg["node"], cfg["elem"], case["fd"])
    ps, pd = _moved(cfg["srcpos"]), _moved(cfg["detpos"])
    if op == "jacobian":
        f = _medium_fields(cfg["node"], np.vstack([ps, pd]), case["fd"])
        J = torch.cat(fem.jacobian(f[:, :len(ps)], f[:, len(ps):]), 1)
        return torch.cat([J.real, J.imag]) if case["fd"] else J
    Bs, Bd = fem.weights(ps), fem.weights(pd)
    B = torch.cat([Bs, Bd], 1)
    if op == "gradient":
        return _exact_gradient(fem, Bs, Bd, *_optical([cfg]), _near([cfg]))

    def forward(prop, per_node):
        p = torch.as_tensor(prop, device="cuda")
        p = p if per_node else p[1]
        phi = fem.solve(fem.matrix(p[..., 0], 1 / (3 * (p[..., 0] + p[..., 1])), per_node), B)
        return Bd.to(phi.dtype).T @ phi[:, :len(ps)], phi

    if op == "forward":
        det, phi = forward(cfg["prop"], case["prop"] == "node")
        return {"det": det, "phi": phi}
    truth = _truth(case, cfg["node"], rng)
    data = forward(truth, True)[0]
    data = data * torch.as_tensor(_noise(tuple(data.shape), case["fd"], rng), device="cuda")
    det, phi = forward(cfg["prop"], True)
    blocks = fem.jacobian(phi[:, :len(ps)], phi[:, len(ps):], case["param"] == "mua")
    J, mis = torch.cat(blocks, 1), (data - det).reshape(-1)
    if case["fd"]:
        J, mis = torch.cat([J.real, J.imag]), torch.cat([mis.real, mis.imag])
    x = _regularised(J, mis, 0.05).cpu().numpy()
    nn, prop = fem.nn, cfg["prop"].copy()
    update = {"mua": x[:nn]}
    d = 1 / (3 * (prop[:, 0] + prop[:, 1]))
    prop[:, 0] += x[:nn]
    if case["param"] != "mua":
        update["dcoeff"] = x[nn:]
        prop[:, 1] = 1 / (3 * (d + x[nn:])) - prop[:, 0]
    return {"resid": np.array([float(mis.abs().sum())]), "prop": prop, "update": update,
            "det": det.cpu().numpy(), "phi": phi.cpu().numpy(),
            "J": J.cpu().numpy() if J.numel() * 4 < 2 ** 31 else None}
