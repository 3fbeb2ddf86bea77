"""Device-resident FEM engine: the layer between the redbirdpy-style dict API
and the CUDA library.

``DeviceMesh`` holds one tetrahedral mesh on the GPU with the structures the
kernels walk (node->tet and node->boundary-face incidence, the CSR pattern,
tet volumes and deldotdel rows), built once by CUDA kernels.  The functions
below run the hot path on device tensors only: assembly, point-optode RHS,
the multi-RHS solve, detector readout and the adjoint Jacobians.  Nothing
here computes on the CPU; every numerical step is a call into
``librbb200.so``.
"""

import ctypes
import threading
import weakref
import zlib

import numpy as np
import torch

from . import _lib
from ._lib import call, ptr, stream

C0 = 299792458000.0  # mm/s (redbirdpy/forward.py:36)


def _dev():
    return _lib.require_cuda()


def _i32(a, device):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.int32), device=device)


def _f64(a, device):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=device)


class DeviceMesh:
    """One mesh on the device.  ``elem``/``face`` are given 1-based (cfg)."""

    def __init__(self, node, elem, face, area, evol=None):
        dev = _dev()
        self.device = dev
        node = np.asarray(node, dtype=np.float64)
        self.nn = int(node.shape[0])
        self.ne = int(elem.shape[0])
        self.node = _f64(node[:, :3], dev)
        with np.errstate(invalid="ignore"):
            self.bbox = (np.nanmin(node[:, :3], axis=0), np.nanmax(node[:, :3], axis=0)) if self.nn else None
        self._coarse = {}
        self._groups = None
        self._mid = False  # not built yet
        self.layout = None  # (positions, bbox, edge, gap) for the groups, where not the nodes' own
        self._edge = None
        if self.ne:
            sel = np.arange(0, self.ne, max(1, self.ne // 65536))
            e = np.asarray(elem)[sel, :2].astype(np.int64) - 1
            if e.min() >= 0 and e.max() < self.nn:
                self._edge = float(np.median(np.linalg.norm(node[e[:, 1], :3] - node[e[:, 0], :3], axis=1)))
        self.elem = _i32(np.asarray(elem)[:, :4].astype(np.int64) - 1, dev)
        face = np.zeros((0, 3), np.int64) if face is None else np.asarray(face)
        self.nf = int(face.shape[0])
        self.face = _i32(face[:, :3].astype(np.int64) - 1, dev) if self.nf else torch.zeros(3, dtype=torch.int32, device=dev)
        self.area = _f64(area, dev) if self.nf else torch.zeros(1, dtype=torch.float64, device=dev)
        st = stream()
        self.eptr, self.elist = self._incidence(self.elem, 4, self.ne, st)
        if self.nf:
            self.fptr, self.flist = self._incidence(self.face, 3, self.nf, st)
        else:
            self.fptr = torch.zeros(self.nn + 1, dtype=torch.int32, device=dev)
            self.flist = torch.zeros(1, dtype=torch.int32, device=dev)
        # CSR pattern
        self.indptr = torch.empty(self.nn + 1, dtype=torch.int32, device=dev)
        wb = _lib.lib().rb_csr_pattern_work_bytes(self.nn)
        work = torch.empty(wb, dtype=torch.uint8, device=dev)
        call("rb_csr_pattern_count", ptr(self.elem), self.nn, ptr(self.eptr), ptr(self.elist),
             ptr(self.indptr), ptr(work), wb, st)
        self.nnz = int(self.indptr[-1].item())
        self.indices = torch.empty(max(self.nnz, 1), dtype=torch.int32, device=dev)
        call("rb_csr_pattern_fill", ptr(self.elem), self.nn, ptr(self.eptr), ptr(self.elist),
             ptr(self.indptr), ptr(self.indices), st)
        rowlen = self.indptr[1:] - self.indptr[:-1]
        self.rmax = int(rowlen.max().item())
        self.emax = int((self.eptr[1:] - self.eptr[:-1]).max().item())
        self.evol_host = evol
        self._ddd = None
        self._evol = None
        self._labels = (None, None)
        self.struct = _lib.RbMesh(
            self.nn, self.ne, self.nf, self.nnz, self.node.data_ptr(), self.elem.data_ptr(),
            self.face.data_ptr(), self.area.data_ptr(), self.eptr.data_ptr(), self.elist.data_ptr(),
            self.fptr.data_ptr(), self.flist.data_ptr(), self.indptr.data_ptr(), self.indices.data_ptr())
        # per-entry contributor tables of the assembly (4*ne + nnz words)
        self.inc_slot = torch.empty(max(4 * self.ne, 1), dtype=torch.int32, device=dev)
        self.slot_mask = torch.empty(max(self.nnz, 1), dtype=torch.int32, device=dev)
        usable = ctypes.c_int32(0)
        call("rb_assembly_tables", ctypes.byref(self.struct), ptr(self.inc_slot), ptr(self.slot_mask),
             ctypes.byref(usable), st)
        if usable.value:
            self.struct.inc_slot = self.inc_slot.data_ptr()
            self.struct.slot_mask = self.slot_mask.data_ptr()
        else:
            self.inc_slot = self.slot_mask = None

    def _incidence(self, cells, nv, ncell, st):
        p = torch.empty(self.nn + 1, dtype=torch.int32, device=self.device)
        lst = torch.empty(max(ncell * nv, 1), dtype=torch.int32, device=self.device)
        wb = _lib.lib().rb_incidence_work_bytes(ncell, nv, self.nn)
        work = torch.empty(wb, dtype=torch.uint8, device=self.device)
        call("rb_incidence", ptr(cells), nv, ncell, self.nn, ptr(p), ptr(lst), ptr(work), wb, st)
        return p, lst

    # -------------------------------------------------------------- geometry
    def _geometry(self):
        self._ddd = torch.empty((self.ne, 10), dtype=torch.float64, device=self.device)
        self._evol = torch.empty(self.ne, dtype=torch.float64, device=self.device)
        call("rb_deldotdel", ptr(self.node), ptr(self.elem), self.ne, ptr(self._ddd), ptr(self._evol), stream())

    @property
    def ddd(self):
        """Ne x 10 deldotdel rows on the device (computed once per mesh)."""
        if self._ddd is None:
            self._geometry()
        return self._ddd

    @property
    def evol(self):
        """Tet volumes on the device: cfg['evol'] when given, else |det|/6."""
        if self._evol is None:
            if self.evol_host is not None:
                self._evol = _f64(self.evol_host, self.device)
            else:
                self._geometry()
        return self._evol

    def labels(self, seg):
        """Device int32 copy of a per-tet label array, uploaded on every call
        into a buffer kept on the mesh (4 bytes per tet: cheaper than a
        checksum of the array, and an array edited in place can never be
        mistaken for the one uploaded before)."""
        a = np.ascontiguousarray(np.asarray(seg).ravel(), dtype=np.int32)
        buf = self._labels[1]
        if buf is None or buf.numel() != a.size:
            buf = torch.empty(a.size, dtype=torch.int32, device=self.device)
            self._labels = (None, buf)
        buf.copy_(torch.from_numpy(a))
        return buf

    def coarse_space(self, target):
        """The CoarseSpace of about ``target`` aggregates (cached per target)."""
        target = int(target)
        if target not in self._coarse:
            self._coarse[target] = CoarseSpace(self, target)
        return self._coarse[target]

    def row_groups(self):
        """The RowGroups of the blocked SpMM (built once), or None when the
        mesh has no usable edge length (e.g. a topology-only mesh)."""
        if self._groups is None:
            edge = self._edge if self.layout is None else self.layout[2]
            if not edge or not np.isfinite(edge) or edge <= 0:
                return None
            self._groups = RowGroups(self, edge)
        return self._groups

    def mid_level(self):
        """The MidLevel of the V-cycle preconditioner (built once), or None
        when the mesh has no row groups, a group has too many neighbours or
        the dense level cannot keep a batch's instances apart."""
        if self._mid is False:
            rg = self.row_groups()
            try:
                self._mid = None if rg is None else MidLevel(self, rg)
            except _lib.RedbirdError as e:
                if e.code != _lib.RB_ESIZE:
                    raise
                self._mid = None
        return self._mid

    def deldotdel_host(self):
        return self.ddd.cpu().numpy()

    def adjacency_host(self):
        """(rows, cols, count) of the off-diagonal pattern, like _femnz
        (utility.py:1020-1041) but with each row's columns ascending."""
        indptr = self.indptr.cpu().numpy().astype(np.int64)
        indices = self.indices[: self.nnz].cpu().numpy().astype(np.int64)
        rows = np.repeat(np.arange(self.nn), np.diff(indptr))
        off = indices != rows
        return rows[off], indices[off], np.diff(indptr) - 1

    def csr_host(self, val):
        """scipy CSR with this pattern and the given device values."""
        from scipy import sparse

        v = val.cpu().numpy()
        return sparse.csr_matrix((v, self.indices[: self.nnz].cpu().numpy(), self.indptr.cpu().numpy()),
                                 shape=(self.nn, self.nn))


def topology_of(elem, nn):
    """A DeviceMesh built from connectivity alone (coordinates zero), enough
    for the Jacobian kernels, which take volumes and deldotdel explicitly.
    Cached by content (shape and a CRC of elem's bytes)."""
    a = np.ascontiguousarray(elem)
    key = (a.shape, a.dtype.str, zlib.crc32(memoryview(a).cast("B")), int(nn))
    if _TOPO.get("key") == key:
        return _TOPO["mesh"]
    m = DeviceMesh(np.zeros((nn, 3)), a, None, None, evol=np.zeros(a.shape[0]))
    _TOPO.update(key=key, mesh=m)
    return m


_TOPO = {}


def _same_arrays(refs, arrays):
    """True when every weak reference still points at the very same object."""
    return len(refs) == len(arrays) and all(
        (r is None and a is None) or (r is not None and r() is a) for r, a in zip(refs, arrays))


def _weak(a):
    if a is None:
        return None
    try:
        return weakref.ref(a)
    except TypeError:  # a list or other non-referenceable container: never reused
        return lambda: object()


def mesh_of(cfg):
    """The DeviceMesh cached in ``cfg['_b200']``, rebuilt when cfg's node,
    elem or face array is replaced by another object.  The cache holds weak
    references to the arrays it was built from, so an array freed and
    replaced by a new one at the same address (same id) is not mistaken for
    it.  Like redbirdpy, which derives face/area/evol/deldotdel from node and
    elem once in meshprep and stores them in cfg, the mesh arrays are taken
    as fixed once prepared: replace them (e.g. run meshprep again) rather
    than edit them in place."""
    arrays = (cfg["node"], cfg["elem"], cfg.get("face"))
    shapes = tuple(np.shape(a) for a in arrays)
    cache = cfg.get("_b200")
    if cache is not None and cache.get("shapes") == shapes and _same_arrays(cache.get("refs", ()), arrays):
        return cache["mesh"]
    m = DeviceMesh(cfg["node"], cfg["elem"], cfg.get("face"), cfg.get("area"), cfg.get("evol"))
    cfg["_b200"] = {"refs": tuple(_weak(a) for a in arrays), "shapes": shapes, "mesh": m}
    return m


# ------------------------------------------------------------ host results
class PinnedPool:
    """Page-locked host buffers for large results copied off the device.  A
    buffer is handed out again only once the numpy array made from it (and
    every view of that array) has been released, so an array returned to the
    caller is never overwritten.  Fresh pageable arrays cost a page fault per
    4 KB on first touch (~2 GB/s); a reused pinned buffer takes the copy at
    PCIe speed (the fields of a 3M-tet frequency-domain reconstruction, 1.07
    GB: 460 -> 20 ms).  At most ``per_shape`` buffers of a shape and
    ``max_bytes`` in all are kept: a new one takes the place of released ones
    of other shapes, and a result that finds no room is copied the plain way.
    Safe to use from several threads; ``trim`` gives released buffers back."""

    def __init__(self, per_shape=3, min_bytes=1 << 20, max_bytes=16 << 30):
        self.per_shape = per_shape
        self.min_bytes = min_bytes
        self.max_bytes = max_bytes
        self._slots = {}  # (shape, dtype) -> [[buffer, weak reference to its array, or None when free]]
        self._lock = threading.Lock()

    def trim(self, need=None):
        """Drop released buffers: all, or until ``need`` more bytes fit."""
        with self._lock:
            return self._trim(need)

    @staticmethod
    def _size(nbytes):
        """What the host allocator takes for a buffer: a power of two."""
        return 1 << max(0, int(nbytes) - 1).bit_length()

    def _bytes(self):
        return sum(self._size(s[0].nbytes) for slots in self._slots.values() for s in slots)

    def _trim(self, need):
        used, dropped = self._bytes(), False
        for key in list(self._slots):
            slots = self._slots[key]
            for slot in list(slots):
                if need is not None and used + need <= self.max_bytes:
                    break
                if slot[1] is None or slot[1]() is None:
                    used -= self._size(slot[0].nbytes)
                    slots.remove(slot)
                    dropped = True
            slot = None
            if not slots:
                del self._slots[key]
        if dropped and hasattr(torch._C, "_host_emptyCache"):
            torch._C._host_emptyCache()  # the buffers go back to the system, not to the host allocator
        return need is None or used + need <= self.max_bytes

    def _take(self, t):
        """A buffer of t's shape reserved for the caller, or None."""
        key = (tuple(t.shape), t.dtype)
        with self._lock:
            slots = self._slots.get(key, [])
            slot = next((s for s in slots if s[1] is None or s[1]() is None), None)
            if slot is None:
                if len(slots) >= self.per_shape or not self._trim(self._size(t.numel() * t.element_size())):
                    return None
                try:
                    slot = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True), None]
                except RuntimeError:  # no page-locked memory to be had
                    return None
                self._slots.setdefault(key, []).append(slot)
            slot[1] = object  # reserved until its array is known (a call gives a live object)
            return slot

    def to_numpy(self, t):
        big = t.numel() * t.element_size() >= self.min_bytes and not t.requires_grad
        slot = self._take(t) if big else None
        if slot is None:
            return t.cpu().numpy()
        try:
            slot[0].copy_(t, non_blocking=True)
            torch.cuda.current_stream(t.device).synchronize()
            arr = slot[0].numpy()
        except BaseException:
            slot[1] = None
            raise
        slot[1] = weakref.ref(arr)
        return arr


host_pool = PinnedPool()


# ------------------------------------------------------------------ optics
class Optics:
    """Per-node or per-tet optical properties on the device, as femlhs reads
    them from cfg['prop'] (redbirdpy/forward.py:126-144)."""

    def __init__(self, mesh, mua, musp, nref, omega, reff):
        dev = mesh.device
        if not isinstance(mua, torch.Tensor):
            mua = np.asarray(mua, dtype=np.float64)
        if len(mua) == mesh.ne:
            self.kind = _lib.RB_PROP_ELEM
        elif len(mua) == mesh.nn:
            self.kind = _lib.RB_PROP_NODE
        else:
            raise ValueError("Property format not recognized")
        self.mua = mua if isinstance(mua, torch.Tensor) else _f64(mua, dev)
        self.musp = musp if isinstance(musp, torch.Tensor) else _f64(musp, dev)
        if isinstance(nref, torch.Tensor) and nref.numel() == len(mua):
            self.nref = nref  # already on the device (kept by the caller across calls)
            self.nref_scalar = 0.0
        elif np.ndim(nref) > 0 and len(nref) == len(mua):
            self.nref = _f64(nref, dev)
            self.nref_scalar = 0.0
        else:
            self.nref = None
            self.nref_scalar = float(np.asarray(nref).ravel()[0]) if np.ndim(nref) > 0 else float(nref)
        self.omega = float(omega)
        self.reff = float(reff)
        self.struct = _lib.RbOptics(self.kind, self.mua.data_ptr(), self.musp.data_ptr(),
                                    None if self.nref is None else self.nref.data_ptr(),
                                    self.nref_scalar, self.omega, self.reff)

    @staticmethod
    def from_cfg(mesh, cfg, mode=1, wv=""):
        """femlhs's property selection (forward.py:105-144): with dicts keyed
        by wavelength, ``prop``, ``reff`` and ``omega`` of wavelength ``wv``."""
        prop = cfg["prop"]
        reff = cfg.get("reff", 0.493)
        omega = cfg.get("omega", 0)
        if isinstance(prop, dict):
            if not wv:
                raise ValueError("per-wavelength properties need a wavelength")
            prop = prop[wv]
            reff = reff[wv] if isinstance(reff, dict) else reff
            omega = omega.get(wv, 0) if isinstance(omega, dict) else omega
        props = np.atleast_2d(np.asarray(prop, dtype=np.float64))
        nn, ne = mesh.nn, mesh.ne
        if props.shape[0] in (nn, ne):
            mua = props[:, 0]
            musp = props[:, 1] * (1 - props[:, 2]) if props.shape[1] >= 3 else props[:, 1]
            nref = props[:, 3] if props.shape[1] >= 4 else 1.37
        elif cfg.get("seg") is not None:
            # label table expanded per tet on the device (prop[seg]); the
            # labels themselves are uploaded once per seg array
            seg = mesh.labels(cfg["seg"])
            nseg = int(seg.numel())
            tab = _f64(props[:, :3] if props.shape[1] >= 3 else props[:, :2], mesh.device)
            mua = torch.empty(nseg, dtype=torch.float64, device=mesh.device)
            musp = torch.empty(nseg, dtype=torch.float64, device=mesh.device)
            call("rb_prop_from_labels", ptr(seg), nseg, ptr(tab), props.shape[0], tab.shape[1], ptr(mua), ptr(musp),
                 stream())
            l0 = int(np.clip(int(np.asarray(cfg["seg"]).ravel()[0]), 0, props.shape[0] - 1))
            nref = props[l0, 3] if props.shape[1] >= 4 else 1.37
        else:
            raise ValueError("Property format not recognized")
        omega = 0.0 if mode == 2 else float(omega or 0)
        return Optics(mesh, mua, musp, nref, omega, reff)


class DeviceMatrix:
    """An assembled FEM matrix in the mesh's CSR pattern (FP64 + FP32 copy)."""

    def __init__(self, mesh, is_complex, val64, val32, dinv64, dinv32):
        self.mesh = mesh
        self.n = mesh.nn
        self.nnz = mesh.nnz
        self.is_complex = bool(is_complex)
        self.val64, self.val32, self.dinv64, self.dinv32 = val64, val32, dinv64, dinv32
        self.indptr, self.indices = mesh.indptr, mesh.indices
        self.struct = _lib.RbCsr(self.n, self.nnz, self.indptr.data_ptr(), self.indices.data_ptr(),
                                 val64.data_ptr(), val32.data_ptr(), dinv64.data_ptr(), dinv32.data_ptr(),
                                 int(self.is_complex))

    @staticmethod
    def from_scipy(A, device=None):
        """Upload a scipy sparse matrix (any square CSR/COO/CSC) for femsolve."""
        from scipy import sparse

        dev = device or _dev()
        A = sparse.csr_matrix(A)
        A.sum_duplicates()
        A.sort_indices()
        cplx = np.iscomplexobj(A.data)

        class _Pattern:
            pass

        pat = _Pattern()
        pat.nn = A.shape[0]
        pat.nnz = A.nnz
        pat.indptr = _i32(A.indptr, dev)
        pat.indices = _i32(A.indices, dev)
        pat.device = dev
        if cplx:
            v64 = torch.as_tensor(np.ascontiguousarray(A.data, dtype=np.complex128), device=dev)
            v32 = torch.empty(A.nnz, dtype=torch.complex64, device=dev)
            d64 = torch.empty(pat.nn, dtype=torch.complex128, device=dev)
            d32 = torch.empty(pat.nn, dtype=torch.complex64, device=dev)
        else:
            v64 = _f64(A.data, dev)
            v32 = torch.empty(A.nnz, dtype=torch.float32, device=dev)
            d64 = torch.empty(pat.nn, dtype=torch.float64, device=dev)
            d32 = torch.empty(pat.nn, dtype=torch.float32, device=dev)
        m = DeviceMatrix(pat, cplx, v64, v32, d64, d32)
        call("rb_csr_prepare", ctypes.byref(m.struct), ptr(v32), ptr(d64), ptr(d32), stream())
        return m


def assemble(mesh, optics, ddd=None, evol=None, tables=True):
    """femlhs on the device -> DeviceMatrix (redbirdpy/forward.py:90-256).
    ``ddd``/``evol`` default to the mesh's own deldotdel rows and volumes;
    ``tables=False`` assembles without the mesh's contributor tables (the
    scan of every incident tet per entry)."""
    dev = mesh.device
    ddd = mesh.ddd if ddd is None else ddd
    evol = mesh.evol if evol is None else evol
    cplx = optics.omega > 0
    t64 = torch.complex128 if cplx else torch.float64
    t32 = torch.complex64 if cplx else torch.float32
    v64 = torch.empty(mesh.nnz, dtype=t64, device=dev)
    v32 = torch.empty(mesh.nnz, dtype=t32, device=dev)
    d64 = torch.empty(mesh.nn, dtype=t64, device=dev)
    d32 = torch.empty(mesh.nn, dtype=t32, device=dev)
    wb = _lib.lib().rb_femlhs_work_bytes(mesh.nn, mesh.ne)
    work = torch.empty(wb, dtype=torch.uint8, device=dev)
    ms = mesh.struct
    if not tables:
        ms = _lib.RbMesh.from_buffer_copy(mesh.struct)
        ms.inc_slot = ms.slot_mask = None
    call("rb_femlhs", ctypes.byref(ms), ctypes.byref(optics.struct), ptr(evol), ptr(ddd), ptr(v64), ptr(v32),
         ptr(d64), ptr(d32), ptr(work), wb, stream())
    return DeviceMatrix(mesh, cplx, v64, v32, d64, d32)


# ------------------------------------------------------------------ optodes
class Optodes:
    """The optodes of one forward model.  Point optodes are located
    (loc int32, -1 outside; bary npts x 4); wide-field patterns (dense nn x
    w columns, cfg['widesrc'] / cfg['widedet']) are kept on the device.
    Right-hand-side columns follow redbirdpy's femrhs order
    (forward.py:278-352): [point src | wide src | point det | wide det];
    ``nsrc`` / ``ndet`` count point and wide ones together."""

    def __init__(self, mesh, pts, nsrc, ndet, wsrc=None, wdet=None):
        dev = mesh.device
        self.npsrc, self.npdet = int(nsrc), int(ndet)
        self.pts_host = np.ascontiguousarray(pts, dtype=np.float64).reshape(-1, 3)
        self.npts = self.pts_host.shape[0]
        self.pts = _f64(self.pts_host, dev) if self.npts else torch.zeros(3, dtype=torch.float64, device=dev)
        self.loc = torch.empty(max(self.npts, 1), dtype=torch.int32, device=dev)
        self.bary = torch.empty((max(self.npts, 1), 4), dtype=torch.float64, device=dev)
        if self.npts:
            call("rb_tsearch", ptr(mesh.node), ptr(mesh.elem), mesh.ne, ptr(self.pts), self.npts, ptr(self.loc),
                 ptr(self.bary), stream())
        self.wsrc = self._patterns(mesh, wsrc)
        self.wdet = self._patterns(mesh, wdet)
        self.nwsrc = 0 if self.wsrc is None else self.wsrc.shape[1]
        self.nwdet = 0 if self.wdet is None else self.wdet.shape[1]
        self.nsrc = self.npsrc + self.nwsrc
        self.ndet = self.npdet + self.nwdet
        self.ncol = self.nsrc + self.ndet

    @staticmethod
    def _patterns(mesh, w):
        if w is None or np.size(w) == 0:
            return None
        w = np.asarray(w, dtype=np.float64)
        if w.ndim == 1:
            w = w[:, None]
        if w.shape[0] != mesh.nn:
            raise ValueError("wide-field patterns must have one row per node (Nn x Npattern)")
        return _f64(w, mesh.device)

    def rhs(self, mesh):
        """Dense nn x ncol real RHS in femrhs's column order."""
        ld = self.ncol
        B = torch.zeros((mesh.nn, ld), dtype=torch.float64, device=mesh.device)
        if self.npsrc:
            call("rb_point_rhs", ptr(mesh.elem), ptr(self.loc), ptr(self.bary), self.npsrc, mesh.nn, ld, 0, ptr(B),
                 stream())
        if self.nwsrc:
            call("rb_wide_rhs", ptr(self.wsrc), mesh.nn, self.nwsrc, self.nwsrc, ld, self.npsrc, ptr(B), stream())
        if self.npdet:
            call("rb_point_rhs", ptr(mesh.elem), ptr(self.loc[self.npsrc:]), ptr(self.bary[self.npsrc:]), self.npdet,
                 mesh.nn, ld, self.nsrc, ptr(B), stream())
        if self.nwdet:
            call("rb_wide_rhs", ptr(self.wdet), mesh.nn, self.nwdet, self.nwdet, ld, self.nsrc + self.npdet, ptr(B),
                 stream())
        return B

    def loc_bary_host(self):
        """loc (1-based float, NaN outside the mesh and for wide-field
        columns) and bary (NaN rows for wide-field), one entry per RHS column
        in femrhs's order (forward.py:298-301)."""
        loc = self.loc[: self.npts].cpu().numpy().astype(np.float64)
        bary = self.bary[: self.npts].cpu().numpy()
        outside = loc < 0
        loc = loc + 1.0
        loc[outside] = np.nan
        if not (self.nwsrc or self.nwdet):
            return loc, bary
        L = np.full(self.ncol, np.nan)
        Bb = np.full((self.ncol, 4), np.nan)
        L[:self.npsrc], Bb[:self.npsrc] = loc[:self.npsrc], bary[:self.npsrc]
        d0 = self.nsrc
        L[d0:d0 + self.npdet], Bb[d0:d0 + self.npdet] = loc[self.npsrc:], bary[self.npsrc:]
        return L, Bb


def locate_optodes(mesh, cfg, wv=""):
    from .utility import getoptodes

    src, det, wsrc, wdet = getoptodes(cfg, wv)
    parts = [p for p in (src, det) if p is not None]
    pts = np.vstack(parts) if parts else np.zeros((0, 3))
    return Optodes(mesh, pts, 0 if src is None else src.shape[0], 0 if det is None else det.shape[0], wsrc, wdet)


def getdet(mesh, opt, phi):
    """detval (ndet x nsrc) = rhs_det^T phi_src (redbirdpy/forward.py:365-442):
    point detector rows by the 4-node barycentric gather, wide-field rows by
    the pattern product over all nodes; columns = point then wide sources."""
    kind = _lib.RB_C128 if phi.is_complex() else _lib.RB_F64
    out = torch.empty((opt.ndet, opt.nsrc), dtype=phi.dtype, device=phi.device)
    if opt.npdet and opt.nsrc:
        call("rb_femgetdet", ptr(mesh.elem), ptr(opt.loc[opt.npsrc:]), ptr(opt.bary[opt.npsrc:]), opt.npdet,
             ptr(phi), phi.shape[1], opt.nsrc, kind, ptr(out), stream())
    if opt.nwdet and opt.nsrc:
        wb = _lib.lib().rb_wide_getdet_work_bytes(opt.nwdet, opt.nsrc, kind)
        work = torch.empty(wb, dtype=torch.uint8, device=phi.device)
        call("rb_wide_getdet", ptr(opt.wdet), mesh.nn, opt.nwdet, opt.nwdet, ptr(phi), phi.shape[1], opt.nsrc, kind,
             ptr(out[opt.npdet:]), ptr(work), wb, stream())
    return out


# -------------------------------------------------------------------- solve
DEFAULT_TOL = 1e-15
COARSE_MAX = 4096      # aggregates the library's coarse solver takes at most
COARSE_MIN_NODES = 20000  # smaller systems converge fast enough on Jacobi alone


def coarse_target(nn, is_complex=False):
    """Default aggregate count of the two-level preconditioner for nn nodes:
    nn / 64 within [256, 2048] for real systems, nn / 128 within [256, 1024]
    for complex ones (their coarse product costs four times as much), never
    above nn / 16.  Measured on the 100 x 100 x 50 mm box at 128 columns
    (forward solve with 1e-4 sweeps, ms; Jacobi alone in brackets): 520k
    nodes CW 2048 aggregates 134, 1183 142 (262); frequency domain 1183 327,
    2048 333 (572); 68k nodes CW 1183 20.1, 2048 26.7 (24.0)."""
    lo, hi, per = (256, 1024, 128) if is_complex else (256, 2048, 64)
    return int(max(1, min(max(lo, min(hi, nn // per)), nn // 16)))


def _finished(dev):
    """Waits for what the current stream has under way: a plan kept on a mesh
    may next be used by another thread on another stream."""
    torch.cuda.current_stream(dev).synchronize()


class CoarseSpace:
    """Aggregates of the two-level preconditioner (``rb_coarse``): the mesh
    nodes binned into cubes of edge h chosen for about ``target`` cubes over
    the bounding box (fewer are nonempty on a mesh that does not fill its
    box).  Built on the device by rb_coarse_aggregate."""

    def __init__(self, mesh, target):
        dev = mesh.device
        nn = mesh.nn
        lo, hi = mesh.bbox
        if not (np.all(np.isfinite(lo)) and np.all(np.isfinite(hi))):
            raise ValueError("coarse space: node coordinates are not finite")
        ext = np.maximum(hi - lo, 0.0)
        span = max(float(ext.max()), 1e-300)
        ext = np.maximum(ext, span * 1e-6)
        h = float(np.cbrt(np.prod(ext) / max(1, min(int(target), COARSE_MAX))))
        self.agg = torch.empty(nn, dtype=torch.int32, device=dev)
        self.agg_ptr = torch.empty(COARSE_MAX + 1, dtype=torch.int32, device=dev)
        self.agg_rows = torch.empty(nn, dtype=torch.int32, device=dev)
        nc = ctypes.c_int64(0)
        for _ in range(64):
            nb = np.maximum(np.ceil(ext / h).astype(np.int64), 1)
            if int(np.prod(nb)) > (1 << 24):
                h *= 1.25
                continue
            wb = _lib.lib().rb_coarse_aggregate_work_bytes(nn, int(np.prod(nb)))
            work = torch.empty(wb, dtype=torch.uint8, device=dev)
            code = _lib.lib().rb_coarse_aggregate(
                ptr(mesh.node), nn, float(lo[0]), float(lo[1]), float(lo[2]), h, int(nb[0]), int(nb[1]), int(nb[2]),
                ptr(self.agg), ptr(self.agg_ptr), ptr(self.agg_rows), ctypes.byref(nc), ptr(work), wb, stream())
            if code == _lib.RB_OK:
                break
            if code != _lib.RB_ESIZE:
                raise _lib.RedbirdError("rb_coarse_aggregate", code, _lib.lib().rb_last_error().decode())
            h *= 1.15
        else:
            raise RuntimeError("coarse space: no bin size found")
        self.nc = int(nc.value)
        self.h = h
        self.nb = tuple(int(v) for v in nb)
        self.struct = _lib.RbCoarse(self.nc, self.agg.data_ptr(), self.agg_ptr.data_ptr(), self.agg_rows.data_ptr())
        _finished(dev)


class RowGroups:
    """Spatial row groups of the blocked SpMM (``rb_rowgroups``): the nodes
    binned into cubes of edge twice the typical edge length (the median length
    of each tet's first edge), origin half an edge below the bounding box, so
    that a structured grid falls into 2 x 2 x 2 blocks; each cube's nodes cut
    into groups of 8; then the column union of every group over the mesh's CSR
    pattern.  Built once per mesh on the device (rb_rowgroups_bin,
    rb_rowgroups_union_*); ``coef`` is the per-solve coefficient scratch."""

    def __init__(self, mesh, edge):
        dev = mesh.device
        nn = mesh.nn
        node, (lo, hi) = (mesh.node, mesh.bbox) if mesh.layout is None else mesh.layout[:2]
        if not (np.isfinite(edge) and edge > 0 and np.all(np.isfinite(lo)) and np.all(np.isfinite(hi))):
            raise ValueError("row groups: degenerate mesh geometry")
        h = 2.0 * edge
        x0 = lo - 0.5 * edge
        ext = np.maximum(hi - x0, 0.0)
        nb = np.maximum(np.ceil(ext / h).astype(np.int64) + 1, 1)
        while int(np.prod(nb)) > (1 << 26):
            h *= 1.25
            nb = np.maximum(np.ceil(ext / h).astype(np.int64) + 1, 1)
        self.rows = torch.empty(8 * nn, dtype=torch.int32, device=dev)
        ng = ctypes.c_int64(0)
        wb = _lib.lib().rb_rowgroups_work_bytes(nn, int(np.prod(nb)))
        work = torch.empty(wb, dtype=torch.uint8, device=dev)
        call("rb_rowgroups_bin", ptr(node), nn, float(x0[0]), float(x0[1]), float(x0[2]), h, int(nb[0]),
             int(nb[1]), int(nb[2]), ptr(self.rows), ctypes.byref(ng), ptr(work), wb, stream())
        self.ng = int(ng.value)
        csr = _lib.RbCsr(nn, mesh.nnz, mesh.indptr.data_ptr(), mesh.indices.data_ptr(), None, None, None, None, 0)
        self.uptr = torch.empty(self.ng + 1, dtype=torch.int32, device=dev)
        wb = _lib.lib().rb_rowgroups_union_work_bytes(self.ng)
        work = torch.empty(wb, dtype=torch.uint8, device=dev)
        nu = ctypes.c_int64(0)
        call("rb_rowgroups_union_count", ctypes.byref(csr), ptr(self.rows), self.ng, ptr(self.uptr),
             ctypes.byref(nu), ptr(work), wb, stream())
        self.nu = int(nu.value)
        self.ucol = torch.empty(max(self.nu, 1), dtype=torch.int32, device=dev)
        self.umask = torch.empty(max(self.nu, 1), dtype=torch.uint8, device=dev)
        call("rb_rowgroups_union_fill", ctypes.byref(csr), ptr(self.rows), self.ng, ptr(self.uptr), ptr(self.ucol),
             ptr(self.umask), stream())
        # coefficient scratch: 8 FP32 values per union entry (real solves)
        self.coef = torch.empty(max(self.nu, 1) * 8, dtype=torch.float32, device=dev)
        self.h = h
        self.struct = _lib.RbRowGroups(self.ng, self.rows.data_ptr(), self.uptr.data_ptr(), self.ucol.data_ptr(),
                                       self.umask.data_ptr(), self.nu, self.coef.data_ptr())
        _finished(dev)


def mid_coarse_target(ng):
    """Default aggregate count of the V-cycle's dense level for ng groups:
    ng / 32 within [64, 1024], never above ng / 8.  Measured (solve, ms; the
    setup grows with the count, the iterations fall): 520k nodes x 128 (67,626
    groups) 256 aggregates 64.4, 726 56.5, 1183 53.8, 2048 53.5; complex 726
    124.0, 1183 112.5, 2048 123.3; 67,626 nodes x 64 (8,788 groups) 256 6.0,
    605 6.6, 1183 7.5; 43,218 x 37 (5,775 groups) 126 4.9, 288 4.9, 600 5.5."""
    return int(max(1, min(max(64, min(1024, ng // 32)), ng // 8)))


class _GroupNodes:
    """What CoarseSpace needs of a mesh, over the row groups: one position
    per group (its first node's)."""

    def __init__(self, mesh, rg):
        node, self.bbox = (mesh.node, mesh.bbox) if mesh.layout is None else mesh.layout[:2]
        self.device, self.nn = mesh.device, rg.ng
        self.node = node[rg.rows[: 8 * rg.ng].view(rg.ng, 8)[:, 0].long()].contiguous()


class MidLevel:
    """The group level of the V-cycle preconditioner (``rb_midlevel``): the
    row groups as aggregates of the nodes, their neighbour pattern, and the
    dense level's aggregates of the groups.  Built once per mesh."""

    def __init__(self, mesh, rg):
        dev = mesh.device
        self.groups = rg
        self.grp = torch.empty(mesh.nn, dtype=torch.int32, device=dev)
        self.mptr = torch.empty(rg.ng + 1, dtype=torch.int32, device=dev)
        wb = _lib.lib().rb_rowgroups_union_work_bytes(rg.ng)
        work = torch.empty(wb, dtype=torch.uint8, device=dev)
        nnz1 = ctypes.c_int64(0)
        call("rb_midlevel_count", ctypes.byref(rg.struct), mesh.nn, ptr(self.grp), ptr(self.mptr),
             ctypes.byref(nnz1), ptr(work), wb, stream())
        self.nnz1 = int(nnz1.value)
        self.mcol = torch.empty(max(self.nnz1, 1), dtype=torch.int32, device=dev)
        call("rb_midlevel_fill", ctypes.byref(rg.struct), ptr(self.grp), ptr(self.mptr), ptr(self.mcol), stream())
        target = mid_coarse_target(rg.ng)
        if mesh.layout is not None:
            # instances side by side leave about half the cells empty; a cell
            # must not reach from one to the next (gap), which takes more of
            # them in a long row of instances
            (lo, hi), gap = mesh.layout[1], mesh.layout[3]
            ext = np.maximum(hi - lo, 1e-6 * float(np.max(hi - lo)))
            target = max(2 * target, int(np.ceil(np.prod(ext) / gap ** 3)))
        self.coarse = CoarseSpace(_GroupNodes(mesh, rg), target)
        if mesh.layout is not None and self.coarse.h > gap:
            raise _lib.RedbirdError("MidLevel", _lib.RB_ESIZE, "cells of the dense level wider than the instances' gap")
        self.struct = _lib.RbMidlevel(ctypes.pointer(rg.struct), self.grp.data_ptr(), self.mptr.data_ptr(),
                                      self.mcol.data_ptr(), self.nnz1, ctypes.pointer(self.coarse.struct))


# Where the V-cycle takes over from the one-launch Jacobi solve (clusters of
# thread blocks, up to 32768 rows): at 450,000 entries of the right-hand side (a
# complex one counts 1.65 times), times 16000 / nodes on smaller meshes, whose
# Jacobi solves need fewer iterations.  One launch / V-cycle in ms: 5814 nodes
# x 128 columns 1.8 / 2.6; 9261 x 48 1.7 / 2.3, x 96 3.2 / 2.7; 12150 x 32 2.2 /
# 2.3, x 64 3.4 / 2.5; 17081 x 16 2.0 / 2.4, x 32 3.0 / 2.4; 24255 x 8 1.2 / 2.4,
# x 16 2.4 / 2.5, x 32 3.6 / 2.6; 32292 x 8 1.5 / 2.6, x 16 3.3 / 2.7; complex
# 7245 x 64 2.0 / 2.9, x 128 3.8 / 3.4; 12150 x 16 1.9 / 2.6, x 32 3.1 / 2.7;
# 17081 x 16 3.5 / 2.9; 24255 x 8 2.2 / 2.9, x 16 4.2 / 3.0; 32292 x 8 2.7 / 3.1.
VCYCLE_ENTRIES = 450000
VCYCLE_NODES = 16000
ONE_LAUNCH_ROWS = 32768


def _one_launch(n, k, cplx):
    """Whether a system of n rows and k columns goes faster in one launch."""
    entries = n * min(k, 128) * (1.65 if cplx else 1.0)
    return n <= ONE_LAUNCH_ROWS and entries * min(1.0, n / VCYCLE_NODES) < VCYCLE_ENTRIES


def _resolve_mid(mat, n, k, prec, coarse, groups, instances, budget):
    """The MidLevel a solve takes, or None: a mixed-precision solve with every
    choice left to the engine ('auto') that is too large for one launch, or of
    stacked instances ('blocks') whose mesh has a layout that keeps their
    groups apart."""
    if groups != "auto" or prec != _lib.RB_MIXED or budget is not None:
        return None
    mesh = getattr(mat, "mesh", None)
    if not hasattr(mesh, "mid_level") or n * (min(k, 128) + 4) >= 2 ** 31:
        return None
    if instances is None:
        take = coarse == "auto" and not _one_launch(n, k, mat.is_complex)
    else:
        take = coarse == "blocks" and n >= COARSE_MIN_NODES and mesh.layout is not None
    return mesh.mid_level() if take else None


def _resolve_groups(mat, groups):
    """RowGroups for solve(groups=...): 'auto' (real matrices assembled on a
    DeviceMesh), a RowGroups, or None/False for the per-row SpMM kernels."""
    if groups is None or groups is False:
        return None
    if isinstance(groups, RowGroups):
        return groups
    mesh = getattr(mat, "mesh", None)
    if groups == "auto":
        if mat.is_complex or not hasattr(mesh, "row_groups"):
            return None
        return mesh.row_groups()
    raise ValueError(f"groups: unsupported value {groups!r}")


def _resolve_coarse(mat, coarse):
    """CoarseSpace for solve(coarse=...): 'auto' (meshes of at least
    COARSE_MIN_NODES nodes), True, an aggregate count, a CoarseSpace, or
    None/False for Jacobi only."""
    if coarse is None or coarse is False or (isinstance(coarse, str) and coarse == "blocks"):
        return None
    if isinstance(coarse, CoarseSpace):
        return coarse
    mesh = getattr(mat, "mesh", None)
    if not hasattr(mesh, "coarse_space"):
        if coarse == "auto":
            return None
        raise ValueError("a coarse space needs a matrix assembled on a DeviceMesh")
    if coarse == "auto":
        return mesh.coarse_space(coarse_target(mat.n, mat.is_complex)) if mat.n >= COARSE_MIN_NODES else None
    if coarse is True:
        return mesh.coarse_space(coarse_target(mat.n, mat.is_complex))
    if isinstance(coarse, (int, np.integer)) and not isinstance(coarse, bool):
        return mesh.coarse_space(int(coarse))
    raise ValueError(f"coarse: unsupported value {coarse!r}")


class Instances:
    """Independent systems stacked block-diagonally (a batch): instance i
    owns rows row_off[i] .. row_off[i+1]-1.  solve(instances=...) then tests
    convergence per (instance, column) and reports each instance's outcome."""

    def __init__(self, row_off, device):
        row_off = np.asarray(row_off, dtype=np.int64)
        if row_off.ndim != 1 or row_off.size < 2 or row_off[0] != 0 or np.any(np.diff(row_off) < 0):
            raise ValueError("instances: row offsets must start at 0 and not decrease")
        self.ninst = row_off.size - 1
        self.n = int(row_off[-1])
        self.row_ptr = torch.as_tensor(row_off, device=device)
        self.row_inst = torch.as_tensor(np.repeat(np.arange(self.ninst, dtype=np.int32), np.diff(row_off)),
                                        device=device)
        self.status = torch.empty(self.ninst, dtype=torch.int32, device=device)

    def struct(self, relres):
        return _lib.RbInstances(self.ninst, self.row_ptr.data_ptr(), self.row_inst.data_ptr(),
                                self.status.data_ptr(), relres.data_ptr())


# per-instance outcome codes of solve(instances=...)
INSTANCE_STATUS = {0: "converged", 1: "iteration cap", 2: "breakdown", 3: "non-finite", 4: "wait gave up"}


class SolveTuner:
    """Autotuner of the solve's launch shapes: for a system it times one
    full solve per candidate (lanes per row of the per-row SpMM, which sets
    the columns a lane takes, and the iterations between host checks) after
    a warm-up, keeps the fastest, and caches it per size bucket (log2 of the
    rows, nonzeros per row, columns, real/complex, precision), so that
    systems of one size share a choice.  The candidates change launch shapes
    only: every candidate computes the same solution."""

    LANES = (0, 8, 16, 32)
    CHECKS = (10, 20)

    def __init__(self):
        self.cache = {}
        self.timings = {}

    @staticmethod
    def bucket(mat, k, kw):
        return (int(np.log2(max(mat.n, 1))), int(round(mat.nnz / max(mat.n, 1))), int(k), bool(mat.is_complex),
                kw.get("precision", "mixed"))

    def options(self, mat, B, **kw):
        """The tuned options for solving mat X = B with solve(**kw)."""
        key = self.bucket(mat, B.shape[1], kw)
        hit = self.cache.get(key)
        if hit is not None:
            return hit
        kw = {k: v for k, v in kw.items() if k not in ("spmm_lanes", "check_every", "profile", "budget")}
        if kw.get("coarse") == "blocks":
            kw["coarse"] = False  # (the shapes are the separate kernels', which fixed budgets run)
        cands = [dict(spmm_lanes=lanes, check_every=c) for lanes in self.LANES for c in self.CHECKS]
        solve(mat, B, **kw, **cands[0])  # warm-up: first launches, plans, caches
        best, times = None, {}
        for cand in cands:
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            _, info = solve(mat, B, **kw, **cand)
            e1.record()
            torch.cuda.synchronize()
            if info["flag"] not in (0, None):
                continue
            ms = e0.elapsed_time(e1)
            times[(cand["spmm_lanes"], cand["check_every"])] = ms
            if best is None or ms < times[(best["spmm_lanes"], best["check_every"])]:
                best = cand
        best = best or cands[0]
        self.cache[key] = best
        self.timings[key] = times
        return best


solve_tuner = SolveTuner()


def _product_kernel(n, k, cplx, prec, form):
    """The kernel of the Krylov product of k columns (the library's dispatch):
    ``form`` 'cycle' (V-cycle), 'one' (one launch), 'groups' (row groups
    given) or 'rows'."""
    if form == "one":
        return "small_solve_kernel"
    pad = (k + 3) // 4 * 4
    if form != "cycle" and (k <= 32 or (k % 2 == 0 and k <= 64)):
        pad = k
    wide, o32 = 64 < pad <= 128, n * pad < 2 ** 31
    if prec == _lib.RB_FP64:
        return "spmm_grp_kernel" if pad in (32, 64, 128) else "spmm_kernel"
    if cplx:
        return "spmm_pair_kernel" if pad == 128 and o32 else "spmm_kernel"
    if wide and form == "cycle":
        return "vc_spmm_kernel"
    if wide and o32:
        return "spmm_blk_kernel" if form == "groups" else "spmm_pair_kernel"
    return "spmm_kernel"


def _add_info(info, inf):
    """One library call's RbSolveInfo into solve's info dict."""
    info["iters"] += inf.iters
    info["outer"] = max(info["outer"], inf.outer)
    info["flag"] = max(info["flag"], inf.flag) if info["flag"] is not None else None
    info["launches"] += inf.launches
    info["sweep_iters_max"] = max(info.get("sweep_iters_max", 0), inf.sweep_iters_max)
    info["relres"] = max(info["relres"], inf.relres)
    for key in ("spmm_ms", "update_ms", "spmm_launches", "update_launches", "coarse_ms", "coarse_launches"):
        info[key] += getattr(inf, key)


def solve(mat, B, precision="mixed", tol=DEFAULT_TOL, inner_tol=None, maxiter=2000, max_outer=10,
          check_every=10, profile=False, x0=None, coarse="auto", groups="auto", instances=None, budget=None,
          spmm_lanes=0):
    """Solve mat X = B for all columns of B (device, nn x k FP64 real).

    Returns (X, info dict).  ``precision='mixed'``: FP32 Jacobi-PCG/COCG
    corrections inside FP64 iterative refinement; ``'fp64'``: the same loop
    entirely in FP64.  Up to 128 columns per library call; wider B is solved
    in column blocks.  ``x0`` (nn x k, the solution's dtype) is an initial
    guess: the refinement starts from its FP64 residual instead of from zero.
    With ``coarse`` and ``groups`` left at 'auto', a mixed-precision solve that
    is too large for one launch (see _one_launch) takes the three-level V-cycle
    preconditioner (MidLevel; a solve that it does not bring to convergence is
    redone with the two-level form, on less than 20000 nodes with Jacobi alone);
    ``coarse='blocks'`` with ``instances`` asks the same of a batch (Jacobi
    alone where it does not apply).  ``coarse`` otherwise adds the aggregation
    coarse space to the Jacobi preconditioner (see _resolve_coarse).
    ``inner_tol`` (relative residual of each FP32 correction sweep) defaults to
    1e-5 with a coarse space and 1e-4 without: on the 520k-node box at 128
    columns, 1e-5 took 3 sweeps / 130 iterations / 113.5 ms against 4 / 150 /
    129.3 ms at 1e-4 and 3 / 150 / 128.6 ms at 1e-6, while Jacobi alone is
    fastest at 1e-4.  ``instances`` (an Instances over the matrix's rows):
    convergence per (instance, column); info then holds ``inst_status``
    (ninst, codes of INSTANCE_STATUS) and ``inst_relres`` (ninst x k).
    ``budget=(sweeps, iterations)``: a fixed budget with no host check or
    read-back (nothing synchronises, so the call can be captured into a CUDA
    graph); columns that converge early turn the rest into no-ops.  It
    needs ``instances`` (one covering all rows is made when None) and no
    coarse space; ``inst_status`` / ``inst_relres`` are then device tensors
    and ``flag`` is None until read.  ``spmm_lanes``: lanes per row of the
    per-row SpMM (0: chosen from the column count; see SolveTuner).  info's
    ``product`` names the kernel of the inner products (last column block),
    ``spmm_kernel`` the same but 'vc_spmm_kernel' for every cycle solve."""
    prec = _lib.RB_FP64 if precision == "fp64" else _lib.RB_MIXED
    n, k = B.shape
    xdt = torch.complex128 if mat.is_complex else torch.float64
    if x0 is not None:
        if tuple(x0.shape) != (n, k):
            raise ValueError("x0 must have the shape of B")
        X = x0.to(device=B.device, dtype=xdt).contiguous().clone()
    else:
        X = torch.empty((n, k), dtype=xdt, device=B.device)
    info = {"iters": 0, "outer": 0, "flag": 0, "launches": 0, "relres": 0.0, "spmm_ms": 0.0, "update_ms": 0.0,
            "spmm_launches": 0, "update_launches": 0, "coarse_ms": 0.0, "coarse_launches": 0}
    if budget is not None:
        max_outer, maxiter = int(budget[0]), int(budget[1])
        check_every = 0
        coarse = False
        if instances is None:
            instances = Instances([0, n], B.device)
    redo = False
    if (coarse == "auto" and groups == "auto" and prec == _lib.RB_MIXED and instances is None and not profile
            and not spmm_lanes and _one_launch(n, k, mat.is_complex)):
        # no coarse space: the library then solves it in one launch; what that
        # does not bring to convergence is redone with the two-level form
        # where the mesh is large enough for one
        redo, coarse = n >= COARSE_MIN_NODES, None
    mid = _resolve_mid(mat, n, k, prec, coarse, groups, instances, budget) if k else None
    cs = _resolve_coarse(mat, coarse) if mid is None else None

    def inner_of(space):
        """The inner tolerance with a coarse space or level (None: without)."""
        t = inner_tol if inner_tol is not None else 1e-5 if space is not None else 1e-4
        return max(tol, 1e-15) if prec == _lib.RB_FP64 and t > 1e-6 else t

    def takes_one_launch(kb):
        """Whether the library solves kb columns in one launch, which reads no row groups."""
        return bool(prec == _lib.RB_MIXED and mid is None and cs is None and instances is None and budget is None
                    and not profile and not spmm_lanes and groups in ("auto", None, False)
                    and _lib.lib().rb_femsolve_one_launch(n, mat.struct.nnz, kb, int(mat.is_complex)))

    rg = None
    if instances is not None and instances.n != n:
        raise ValueError("instances do not cover the matrix's rows")
    opts = _lib.RbSolveOpts(prec, int(max_outer), int(maxiter), int(check_every), float(tol),
                            float(inner_of(mid if mid is not None else cs)), int(bool(profile)), int(x0 is not None),
                            ctypes.pointer(cs.struct) if cs is not None else None, None, None, int(spmm_lanes),
                            int(redo))
    inst_status, inst_relres = [], []
    for c0 in range(0, k, 128):
        kb = min(128, k - c0)
        if instances is not None:
            rel = torch.empty((instances.ninst, kb), dtype=torch.float64, device=B.device)
            ist = instances.struct(rel)
            opts.instances = ctypes.pointer(ist)
        Bb = B[:, c0:c0 + kb].contiguous() if (c0 or kb != k) else B
        if c0 or kb != k:
            Xb = X[:, c0:c0 + kb].contiguous() if x0 is not None else torch.empty((n, kb), dtype=xdt, device=B.device)
        else:
            Xb = X
        inf = _lib.RbSolveInfo()
        if mid is not None:
            wb = _lib.lib().rb_femsolve_mid_work_bytes(ctypes.byref(mat.struct), ctypes.byref(mid.struct), kb)
            if instances is not None:
                wb += _lib.lib().rb_instances_work_bytes(instances.ninst, (kb + 3) // 4 * 4)
            try:
                work = torch.empty(wb, dtype=torch.uint8, device=B.device)
            except torch.cuda.OutOfMemoryError:
                work = None  # the two-level form needs a fifth less
            if work is not None:
                try:
                    call("rb_femsolve_mid", ctypes.byref(mat.struct), ctypes.byref(mid.struct), ptr(Bb), ptr(Xb), kb,
                         ctypes.byref(opts), ctypes.byref(inf), ptr(work), wb, stream())
                except _lib.RedbirdError as e:
                    if e.code != _lib.RB_EBREAKDOWN:  # (a zero or non-finite pivot of the dense level)
                        raise
                    work = None
            if work is None or inf.flag != 0:
                # the cycle assumes a definite operator (positive diagonal,
                # real part); what it does not solve gets the two-level form
                work = None
                cs = _resolve_coarse(mat, coarse)
                opts.coarse = ctypes.pointer(cs.struct) if cs is not None else None
                opts.inner_tol = float(inner_of(cs))
                mid = None
                if x0 is not None:
                    Xb.copy_(x0[:, c0:c0 + kb])
        if mid is not None:
            if Xb is not X:
                X[:, c0:c0 + kb] = Xb
            _add_info(info, inf)
            if instances is not None:
                inst_status.append(instances.status.cpu().numpy())
                inst_relres.append(rel)
            continue
        while True:
            if prec == _lib.RB_MIXED:
                one = takes_one_launch(kb)
                rg = rg if one or rg is not None else _resolve_groups(mat, groups)
                opts.groups = ctypes.pointer(rg.struct) if rg is not None and not one else None
            wb = _lib.lib().rb_femsolve_work_bytes(n, mat.struct.nnz, kb, int(mat.is_complex), prec)
            if cs is not None:
                wb += _lib.lib().rb_coarse_work_bytes(cs.nc, kb, int(mat.is_complex), prec)
            if instances is not None:
                wb += _lib.lib().rb_instances_work_bytes(instances.ninst, kb)
            work = torch.empty(wb, dtype=torch.uint8, device=B.device)
            call("rb_femsolve", ctypes.byref(mat.struct), ptr(Bb), ptr(Xb), kb, ctypes.byref(opts), ctypes.byref(inf),
                 ptr(work), wb, stream())
            if inf.flag == 0 or not redo:
                break
            redo, cs = False, _resolve_coarse(mat, "auto")
            if cs is None:
                break
            opts.coarse = ctypes.pointer(cs.struct)
            opts.inner_tol = float(inner_of(cs))
            if x0 is not None:
                Xb.copy_(x0[:, c0:c0 + kb])
        if Xb is not X:
            X[:, c0:c0 + kb] = Xb
        _add_info(info, inf)
        if instances is not None:
            inst_status.append(instances.status.clone() if budget is not None else instances.status.cpu().numpy())
            inst_relres.append(rel)
    if instances is not None and budget is not None:
        info["flag"] = None
        info["relres"] = None
        info["inst_status"] = torch.amax(torch.stack(inst_status), dim=0) if len(inst_status) > 1 else inst_status[0]
        info["inst_relres"] = torch.cat(inst_relres, dim=1) if len(inst_relres) > 1 else inst_relres[0]
    elif instances is not None:
        info["inst_status"] = np.max(np.stack(inst_status), axis=0)
        info["inst_relres"] = torch.cat(inst_relres, dim=1).cpu().numpy()
    info["coarse_nc"] = mid.coarse.nc if mid is not None else cs.nc if cs is not None else 0
    # the inner product of the last column block
    kb = k - 128 * ((k - 1) // 128) if k else 0
    form = "cycle" if mid is not None else "one" if k and prec == _lib.RB_MIXED and one else "groups" if rg else "rows"
    info["product"] = _product_kernel(n, kb, mat.is_complex, prec, form)
    # (a cycle solve's products go by one name here, whichever kernel fits the width)
    info["spmm_kernel"] = "vc_spmm_kernel" if mid is not None else info["product"]
    return X, info


# ----------------------------------------------------------------- Jacobian
def pair_map(sd, nsrc_cols=None):
    """Column map of the active (src, det) pairs of an sd table for rb_jac:
    (cols, det0, ndet, pair_src, pair_det, src_col, det_col)."""
    sd = np.asarray(sd)
    act = sd[sd[:, 2] == 1, :2] if sd.shape[1] >= 3 else sd[:, :2]
    act = act.astype(np.int64)
    s_u = np.unique(act[:, 0])
    d_u = np.unique(act[:, 1])
    cols = np.concatenate([s_u, d_u])
    psrc = np.searchsorted(s_u, act[:, 0])
    pdet = np.searchsorted(d_u, act[:, 1])
    return cols, len(s_u), len(d_u), psrc, pdet, act[:, 0], act[:, 1]


def _grid_nsd(psrc, pdet, nsu, ndet, mult=4):
    """nsd as rb_jac expects it: negative when the pairs are every (source,
    detector) combination in detector-major order (sdmap's layout) with both
    counts multiples of 4, which selects the register-blocked kernel path;
    mult=1 for rb_jac_multi, which takes any counts."""
    nsd = len(psrc)
    if (nsd == nsu * ndet and nsu % mult == 0 and ndet % mult == 0
            and np.array_equal(psrc, np.tile(np.arange(nsu), ndet))
            and np.array_equal(pdet, np.repeat(np.arange(ndet), nsu))):
        return -nsd
    return nsd


_PAIRS = {}


def _pair_dev(sd, dev):
    """pair_map of ``sd`` with its three index arrays on the device, cached
    by content (a loop over one sd table uploads them once)."""
    a = np.ascontiguousarray(sd)
    key = (a.shape, a.dtype.str, zlib.crc32(memoryview(a).cast("B")), str(dev))
    hit = _PAIRS.get(key)
    if hit is None:
        cols, det0, ndet, psrc, pdet, _, _ = pair_map(a)
        hit = (cols, det0, ndet, psrc, pdet, _i32(cols, dev), _i32(psrc, dev), _i32(pdet, dev),
               _grid_nsd(psrc, pdet, det0, ndet))
        if len(_PAIRS) > 64:
            _PAIRS.clear()
        _PAIRS[key] = hit
    return hit


def jac_tensor_cores(on=True):
    """Allow or forbid (the default) the tensor-core pair products of rb_jac."""
    call("rb_jac_tensor_cores", int(bool(on)))


def _jac_checked():
    """The outcome of the tensor-core Jacobian launches so far (synchronises;
    skipped while a CUDA graph is being captured)."""
    if not torch.cuda.is_current_stream_capturing():
        call("rb_jac_status", stream())


def jacobian(mesh, phi, sd, what="mua", out_dtype=torch.float32, J=None, ldj=None, evol=None, ddd=None):
    """Adjoint Jacobian rows on the device (nsd x nn), see rb_jac.
    what: 'mua' (reference semantics, forward.py:509-569), 'mua_nodal'
    (exact for node-based properties at fixed D) or 'D'."""
    dev = phi.device
    cols, det0, ndet, psrc, pdet, colsd, ps, pd, gnsd = _pair_dev(sd, dev)
    nsd = len(psrc)
    cplx = phi.is_complex()
    if cplx and not out_dtype.is_complex:
        out_dtype = torch.complex64 if out_dtype == torch.float32 else torch.complex128
    if J is None:
        J = torch.empty((nsd, mesh.nn), dtype=out_dtype, device=dev)
        ldj = mesh.nn
    phi_kind = {torch.float64: _lib.RB_F64, torch.complex128: _lib.RB_C128, torch.float32: _lib.RB_F32,
                torch.complex64: _lib.RB_C64}[phi.dtype]
    out_kind = {torch.float64: _lib.RB_F64, torch.complex128: _lib.RB_C128, torch.float32: _lib.RB_F32,
                torch.complex64: _lib.RB_C64}[J.dtype]
    w = {"mua": _lib.RB_JAC_MUA_REF, "mua_nodal": _lib.RB_JAC_MUA_NODAL, "D": _lib.RB_JAC_D}[what]
    ev = evol if evol is not None else mesh.evol
    dd = ddd if ddd is not None else (mesh.ddd if w == _lib.RB_JAC_D else None)
    # pair groups: at most 128 staged columns / 64 detectors per launch
    if len(cols) > 128 or ndet > 64:
        raise ValueError("rb_jac stages at most 128 phi columns and 64 detectors per call")
    call("rb_jac", ctypes.byref(mesh.struct), w, ptr(phi), phi_kind, phi.shape[1], ptr(colsd), len(cols), det0, ndet,
         ptr(ps), ptr(pd), gnsd, ptr(J), ldj, out_kind, mesh.rmax, mesh.emax, ptr(ev), ptr(dd), stream())
    if J.dtype in (torch.float32, torch.complex64):
        _jac_checked()
    return J


def jacobian_elem(mesh, phi, sd, evol=None):
    _, _, _, _, _, scol, dcol = pair_map(sd)
    nsd = len(scol)
    Je = torch.empty((nsd, mesh.ne), dtype=phi.dtype, device=phi.device)
    kind = _lib.RB_C128 if phi.is_complex() else _lib.RB_F64
    ev = evol if evol is not None else mesh.evol
    sc, dc = _i32(scol, phi.device), _i32(dcol, phi.device)  # kept alive across the launch
    call("rb_jac_elem", ctypes.byref(mesh.struct), ptr(ev), ptr(phi), kind, phi.shape[1], ptr(sc), ptr(dc), nsd,
         ptr(Je), stream())
    return Je


def jacobian_grad(mesh, phi, lam, ns, mua=True, dcoef=True):
    """(gm, gd): sums over the column pairs (phi[:, s], lam[:, s]), s < ns, of
    the exact node-based rows 'mua_nodal' and 'D' (real parts), one pass over
    the tets without forming a row (rb_jac_grad); None for one not asked."""
    if ns > 64:
        raise ValueError("jacobian_grad: at most 64 column pairs per call")
    phi, lam = phi.contiguous(), lam.contiguous()
    kind = _lib.RB_C128 if phi.is_complex() else _lib.RB_F64
    gm = torch.empty(mesh.nn, dtype=torch.float64, device=phi.device) if mua else None
    gd = torch.empty(mesh.nn, dtype=torch.float64, device=phi.device) if dcoef else None
    wb = _lib.lib().rb_jac_grad_work_bytes(mesh.ne)
    work = torch.empty(wb, dtype=torch.uint8, device=phi.device)
    call("rb_jac_grad", ctypes.byref(mesh.struct), ptr(phi), phi.shape[1], ptr(lam), lam.shape[1], ns, kind,
         ptr(mesh.evol), ptr(mesh.ddd if dcoef else None), ptr(gm), ptr(gd), ptr(work), wb, stream())
    return gm, gd


# ------------------------------------------------------------ Gauss-Newton
def _pad4(n):
    return (n + 3) // 4 * 4


def _pad8(n):
    return (n + 7) // 8 * 8


def _jac_what(name, mode):
    """The RB_JAC_* quantity of a GN parameter."""
    if name == "mua":
        return _lib.RB_JAC_MUA_REF if mode == "reference" else _lib.RB_JAC_MUA_NODAL
    if name == "D":
        return _lib.RB_JAC_D
    raise ValueError(f"unknown parameter {name}")


# Nodes from which the full grid's rows take the pipelined kernel (and its
# workspace): 16 x 16 pairs, one quantity, general kernel / this, ms: 2002 nodes
# 0.181 / 0.179 (64 x 64 0.350 / 0.394), 16,926 nodes 0.352 / 0.279 (0.917 / 0.782),
# 58,609 nodes 0.869 / 0.593 (2.291 / 1.986)
JAC_GRID_NODES = 8192


def _jac_grid_bytes(mesh, phi, det0, ndet, psrc, pdet, acc64, count):
    """Workspace of the pipelined kernel (rb_jac_multi) for rows over ``count``
    nodes, 0 where the general kernel forms them."""
    if not acc64 or count < JAC_GRID_NODES or phi.dtype not in (torch.float64, torch.complex128):
        return 0
    cplx = int(phi.is_complex())
    if not _lib.lib().rb_jac_multi_wins(mesh.rmax, mesh.emax, det0, ndet, cplx):
        return 0
    if _grid_nsd(psrc, pdet, det0, ndet, 1) >= 0:
        return 0
    return _lib.lib().rb_jac_multi_work_bytes(mesh.rmax, det0, ndet, cplx)


def _jac_params(mesh, whats, phi, phi_kind, colsd, nc, det0, ndet, ps, pd, gnsd, wb, J, ldj, out_kind, stride, node0,
                count):
    """The rows of every parameter, parameter p's columns from p * stride, by
    the pipelined kernel with wb bytes of workspace (the full grid) or, wb = 0,
    by the general one."""
    if wb and whats:
        npar = len(whats)
        work = torch.empty(wb, dtype=torch.uint8, device=phi.device)
        need_ddd = _lib.RB_JAC_D in whats
        call("rb_jac_multi", ctypes.byref(mesh.struct), npar, (ctypes.c_int32 * npar)(*whats),
             (ctypes.c_int64 * npar)(*(p * stride for p in range(npar))), ptr(phi), phi_kind, phi.shape[1], ptr(colsd),
             nc, det0, ndet, ptr(ps), ptr(pd), -abs(gnsd), ptr(J), ldj, out_kind, mesh.rmax, mesh.emax, ptr(mesh.evol),
             ptr(mesh.ddd if need_ddd else None), node0, count, ptr(work), wb, stream())
        return
    m, f, c, s, d, v, st = (ctypes.byref(mesh.struct), ptr(phi), ptr(colsd), ptr(ps), ptr(pd), ptr(mesh.evol), stream())
    for p, w in enumerate(whats):
        call("rb_jac_range", m, w, f, phi_kind, phi.shape[1], c, nc, det0, ndet, s, d, gnsd, ptr(J[:, p * stride:]), ldj,
             out_kind, mesh.rmax, mesh.emax, v, ptr(mesh.ddd if w == _lib.RB_JAC_D else None), node0, count, st)


def jacobian_matrix(mesh, phi, sd, params=("mua",), mode="reference", dtype=torch.float32, acc64=False):
    """The real Jacobian of the GN step (FP32, or BF16 with ``dtype``), rows x
    columns = (nsd or 2 nsd) x (len(params) * nn), stored with a row stride
    padded to 16 bytes (32, a whole sector, where the pipelined kernel writes them).
    Complex fields give matreform 'real' stacking [Re; Im] (recon.py:532-546).
    mode 'reference' = redbirdpy's jac for mua (forward.py:509-569);
    'exact' = derivatives of the node-based assembly ('mua' at fixed D, 'D').
    ``acc64``: FP32 rows whose products are formed in FP64 (only the storage
    rounds: ~6e-8 relative per entry instead of ~3e-7)."""
    cols, det0, ndet, psrc, pdet, _, _ = pair_map(sd)
    nsd = len(psrc)
    cplx = phi.is_complex()
    rows = 2 * nsd if cplx else nsd
    nn = mesh.nn
    bf = dtype == torch.bfloat16
    wb = _jac_grid_bytes(mesh, phi, det0, ndet, psrc, pdet, acc64 and not bf, nn)
    ldj = _pad8(len(params) * nn) if bf or wb else _pad4(len(params) * nn)
    # every column below len(params) * nn is written by rb_jac; only the
    # row padding (read by the gram's aligned tiles) is cleared here
    J = torch.empty((rows, ldj), dtype=dtype, device=phi.device)
    if ldj > len(params) * nn:
        J[:, len(params) * nn:].zero_()
    if bf:
        out_kind = _lib.RB_JAC_SPLIT_BF16 if cplx else _lib.RB_JAC_BF16
    elif acc64:
        out_kind = _lib.RB_JAC_SPLIT_F32_ACC64 if cplx else _lib.RB_JAC_F32_ACC64
    else:
        out_kind = _lib.RB_JAC_SPLIT_F32 if cplx else _lib.RB_F32
    phi_kind = {torch.float64: _lib.RB_F64, torch.complex128: _lib.RB_C128, torch.float32: _lib.RB_F32,
                torch.complex64: _lib.RB_C64}[phi.dtype]
    colsd, ps, pd = _i32(np.concatenate([cols, psrc, pdet]), phi.device).split([len(cols), nsd, nsd])  # one upload
    _jac_params(mesh, [_jac_what(name, mode) for name in params], phi, phi_kind, colsd, len(cols), det0, ndet, ps, pd,
                nsd if wb else _grid_nsd(psrc, pdet, det0, ndet), wb, J, ldj, out_kind, nn, 0, nn)
    _jac_checked()
    return J, len(params) * nn


def sumsq(J, K):
    out = torch.empty(1, dtype=torch.float64, device=J.device)
    wb = _lib.lib().rb_sumsq_work_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=J.device)
    fn = "rb_sumsq_bf16" if J.dtype == torch.bfloat16 else "rb_sumsq"
    call(fn, ptr(J), J.shape[0], K, J.shape[1], ptr(out), ptr(work), wb, stream())
    return out


def row_sumsq(J, K, bf16_copy=False):
    """(rows, total): FP64 sums of squares of J's rows (the exact diagonal of
    J J^T for the stored rows) and their sum (the Frobenius sum), one pass.
    ``bf16_copy`` (FP32 J): the same pass also returns J rounded to BF16
    (rows, total, Jb), the operand of a BF16 product whose refinement runs
    over the FP32 rows."""
    M = J.shape[0]
    rows = torch.empty(M, dtype=torch.float64, device=J.device)
    total = torch.empty(1, dtype=torch.float64, device=J.device)
    if bf16_copy:
        if J.dtype != torch.float32:
            raise ValueError("a BF16 copy is made from FP32 rows")
        Jb = torch.empty((M, _pad8(K)), dtype=torch.bfloat16, device=J.device)
        call("rb_row_sumsq_to_bf16", ptr(J), M, K, J.shape[1], ptr(rows), ptr(total), ptr(Jb), Jb.shape[1],
             stream())
        return rows, total, Jb
    fn = "rb_row_sumsq_bf16" if J.dtype == torch.bfloat16 else "rb_row_sumsq"
    call(fn, ptr(J), M, K, J.shape[1], ptr(rows), ptr(total), stream())
    return rows, total


def gram(J, K, alpha=1.0, precision="tf32"):
    """H = alpha J J^T (M x M FP64) on the tensor cores.  precision 'tf32'
    (one pass) or 'tf32x3' (split hi/lo, three passes; J is left as hi and
    the returned lo completes it); a BF16 J takes the BF16 MMA, and so does
    'bf16' with FP32 rows (on a BF16 copy of them)."""
    if precision == "bf16" and J.dtype == torch.float32:  # the product from a BF16 copy
        J = row_sumsq(J, K, bf16_copy=True)[2]
    M, ldj = J.shape
    H = torch.empty((M, M), dtype=torch.float64, device=J.device)
    lo = None
    wb = _lib.lib().rb_gram_work_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=J.device)
    bf16 = J.dtype == torch.bfloat16
    if not bf16:
        if precision == "tf32x3":
            lo = torch.empty_like(J)
            call("rb_split_tf32", ptr(J), ptr(lo), M, K, ldj, stream())
        elif precision != "tf32":
            raise ValueError(f"unknown gram precision {precision}")
    # long rows: the products are formed from compact copies of J's column
    # slabs (same result; 2x faster slabs at a row stride of megabytes)
    sb = _lib.lib().rb_gram_stage_bytes(M, K, ldj, 2 if bf16 else 4, int(lo is not None))
    stage = torch.empty(sb, dtype=torch.uint8, device=J.device) if sb else None
    sp = ptr(stage) if stage is not None else None
    if bf16:
        call("rb_gram_bf16_staged", ptr(J), M, K, ldj, float(alpha), ptr(H), M, sp, sb, ptr(work), wb, stream())
    else:
        call("rb_gram_staged", ptr(J), ptr(lo), M, K, ldj, float(alpha), ptr(H), M, sp, sb, ptr(work), wb,
             stream())
    return H, lo


def gemv_n(J, K, x, alpha=1.0, beta=0.0, out=None, lo=None):
    """out = alpha J x + beta out on the device (J FP32 / BF16 rows, x FP64
    K-vector); with ``lo`` the split remainder of J is added as well."""
    M, ldj = J.shape
    if out is None:
        out = torch.empty(M, dtype=torch.float64, device=J.device)
    fn = "rb_gemv_n_bf16" if J.dtype == torch.bfloat16 else "rb_gemv_n"
    wb = _lib.lib().rb_gemv_n_work_bytes(M, K)
    work = torch.empty(wb, dtype=torch.uint8, device=J.device)
    call(fn, ptr(J), M, K, ldj, ptr(x), float(alpha), float(beta), ptr(out), ptr(work), wb, stream())
    if lo is not None:
        call("rb_gemv_n", ptr(lo), M, K, ldj, ptr(x), float(alpha), 1.0, ptr(out), ptr(work), wb, stream())
    return out


def norm2(x):
    """||x||_2 of an FP64 device vector (rb_dot), as a Python float."""
    out = torch.empty(1, dtype=torch.float64, device=x.device)
    wb = _lib.lib().rb_dot_work_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=x.device)
    call("rb_dot", x.numel(), ptr(x), ptr(x), ptr(out), ptr(work), wb, stream())
    return float(out.item()) ** 0.5


def normal_factor(J, K, lam, alpha=1.0, precision="tf32", lam_rel=None, rowsq=None, Jb=None):
    """The tensor-core half of reginvunder (recon.py:474-483): H = alpha J J^T
    (+ lam I, lam relative to the largest diagonal entry with ``lam_rel``),
    unit-diagonal normalisation (_normalize_diag, recon.py:784-789), FP64
    Cholesky in place.  ``rowsq`` (row_sumsq's rows) replaces the product's
    diagonal by the exact one, so that a relative lam and the normalisation
    carry no tensor-core input rounding.  ``Jb`` (J rounded to BF16, from
    row_sumsq) is the product's operand when given: a BF16 factor of the
    FP32 rows' system, which normal_solve then refines over those rows.
    Returns (H, di, lo, lam)."""
    M, ldj = J.shape
    dev = J.device
    H, lo = gram(Jb if Jb is not None else J, K, alpha, precision)
    if rowsq is not None:
        call("rb_set_diag", ptr(H), M, M, ptr(rowsq), float(alpha), stream())
    if lam_rel is not None:
        lam = float(lam_rel) * float(H.diagonal().max().item())
    di = torch.empty(M, dtype=torch.float64, device=dev)
    call("rb_reginv_prepare", ptr(H), M, M, float(lam), ptr(di), stream())
    wb = _lib.lib().rb_cholesky_work_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=dev)
    call("rb_cholesky", ptr(H), M, M, ptr(work), wb, stream())
    return H, di, lo, float(lam)


class StoredJacobian:
    """The passes normal_solve makes over a J held in HBM (FP32 or BF16
    rows; ``lo`` the split remainder of a tf32x3 factorisation)."""

    def __init__(self, J, K, lo=None):
        self.J, self.K, self.lo = J, K, lo
        self.rows = J.shape[0]

    def jt(self, y, alpha=1.0):
        return gemv_t(self.J, self.K, y, alpha, lo=self.lo)

    def jt_then_j(self, y):
        """(u, J u) with u = J^T y: two passes over J."""
        u = gemv_t(self.J, self.K, y, 1.0, lo=self.lo)
        return u, gemv_n(self.J, self.K, u, 1.0, 0.0, lo=self.lo)


class SlabJacobian:
    """The GN matrix J = [J_p1 | J_p2 ...] (rows x K, K = len(params) * nn)
    never held whole, for meshes whose Jacobian does not fit in HBM: node
    slabs of ``width`` columns per parameter are recomputed from the stored
    fields (rb_jac_range, redbirdpy's jac in column blocks,
    forward.py:509-569) on every pass, so a pass costs one Jacobian build
    and the memory is rows x len(params) x width.  Offers the same passes as
    StoredJacobian plus the Frobenius sum and the tensor-core product."""

    def __init__(self, mesh, phi, sd, params=("mua",), mode="reference", width=4096, dtype=torch.float32,
                 acc64=False):
        self.mesh, self.phi, self.params, self.dtype = mesh, phi, tuple(params), dtype
        self.cols, self.det0, self.ndet, psrc, pdet, self.colsd, self.ps, self.pd, self.gnsd = _pair_dev(sd, phi.device)
        if len(self.cols) > 128 or self.ndet > 64:
            raise ValueError("rb_jac stages at most 128 phi columns and 64 detectors per call")
        nsd = len(psrc)
        self.cplx = phi.is_complex()
        self.rows = 2 * nsd if self.cplx else nsd
        self.nn = mesh.nn
        self.K = len(self.params) * self.nn
        self.width = int(max(1, min(width, self.nn)))
        self.bf = dtype == torch.bfloat16
        self.wb = _jac_grid_bytes(mesh, phi, self.det0, self.ndet, psrc, pdet, acc64 and not self.bf, self.width)
        pad = self._pad = _pad8 if self.bf or self.wb else _pad4
        self.buf = torch.empty(self.rows * pad(len(self.params) * self.width), dtype=dtype, device=phi.device)
        if self.bf:
            self.out_kind = _lib.RB_JAC_SPLIT_BF16 if self.cplx else _lib.RB_JAC_BF16
        elif acc64:
            self.out_kind = _lib.RB_JAC_SPLIT_F32_ACC64 if self.cplx else _lib.RB_JAC_F32_ACC64
        else:
            self.out_kind = _lib.RB_JAC_SPLIT_F32 if self.cplx else _lib.RB_F32
        self.phi_kind = {torch.float64: _lib.RB_F64, torch.complex128: _lib.RB_C128, torch.float32: _lib.RB_F32,
                         torch.complex64: _lib.RB_C64}[phi.dtype]
        self.whats = [_jac_what(name, mode) for name in self.params]
        self.passes = 0

    def ranges(self):
        for a in range(0, self.nn, self.width):
            yield a, min(self.nn, a + self.width)

    def slab(self, a, b):
        """J restricted to nodes a..b-1 (every parameter), rows x pad(P c),
        columns [p1 nodes a..b-1 | p2 nodes a..b-1 ...]; the buffer is reused."""
        c = b - a
        ks = len(self.params) * c
        ld = self._pad(ks)
        Js = self.buf[: self.rows * ld].view(self.rows, ld)
        if ld > ks:
            Js[:, ks:].zero_()
        _jac_params(self.mesh, self.whats, self.phi, self.phi_kind, self.colsd, len(self.cols), self.det0, self.ndet,
                    self.ps, self.pd, self.gnsd, self.wb if c >= JAC_GRID_NODES else 0, Js, ld, self.out_kind, c, a, c)
        _jac_checked()
        return Js, ks

    def _pieces(self, a, b):
        """K-space slices of a slab's columns, in the slab's column order."""
        return [slice(p * self.nn + a, p * self.nn + b) for p in range(len(self.params))]

    def row_sumsq(self):
        """(rows, total) as engine.row_sumsq, summed over the slabs."""
        rows = torch.zeros(self.rows, dtype=torch.float64, device=self.phi.device)
        tot = torch.zeros(1, dtype=torch.float64, device=self.phi.device)
        for a, b in self.ranges():
            Js, ks = self.slab(a, b)
            r_s, t_s = row_sumsq(Js, ks)
            call("rb_axpby", self.rows, 1.0, ptr(r_s), 1.0, ptr(rows), stream())
            call("rb_axpby", 1, 1.0, ptr(t_s), 1.0, ptr(tot), stream())
        self.passes += 1
        return rows, tot

    def sumsq(self):
        return self.row_sumsq()[1]

    def gram(self, alpha=1.0, precision="tf32"):
        """H = alpha sum over slabs of J_s J_s^T (FP64 accumulation of the
        tensor-core products of each slab; 'bf16' with FP32 slabs forms the
        product from a BF16 copy of each slab)."""
        M = self.rows
        H = torch.zeros((M, M), dtype=torch.float64, device=self.phi.device)
        for a, b in self.ranges():
            Js, ks = self.slab(a, b)
            Hs, _ = gram(Js, ks, alpha, precision)
            call("rb_axpby", M * M, 1.0, ptr(Hs), 1.0, ptr(H), stream())
        self.passes += 1
        return H

    def jt(self, y, alpha=1.0):
        out = torch.empty(self.K, dtype=torch.float64, device=self.phi.device)
        for a, b in self.ranges():
            Js, ks = self.slab(a, b)
            us = gemv_t(Js, ks, y, alpha)
            c = b - a
            for p, sl in enumerate(self._pieces(a, b)):
                out[sl] = us[p * c:(p + 1) * c]
        self.passes += 1
        return out

    def jt_then_j(self, y):
        """(u, J u) with u = J^T y in one pass: per slab u_s = J_s^T y, then
        the slab's share J_s u_s while J_s is still in HBM."""
        M = self.rows
        u = torch.empty(self.K, dtype=torch.float64, device=self.phi.device)
        Ju = torch.zeros(M, dtype=torch.float64, device=self.phi.device)
        for a, b in self.ranges():
            Js, ks = self.slab(a, b)
            us = gemv_t(Js, ks, y, 1.0)
            gemv_n(Js, ks, us, 1.0, 1.0, out=Ju)
            c = b - a
            for p, sl in enumerate(self._pieces(a, b)):
                u[sl] = us[p * c:(p + 1) * c]
        self.passes += 1
        return u, Ju


def normal_factor_op(op, lam, alpha=1.0, precision="tf32", lam_rel=None, rowsq=None):
    """normal_factor for a SlabJacobian: the product summed over its slabs."""
    M = op.rows
    dev = op.phi.device
    H = op.gram(alpha, precision)
    if rowsq is not None:
        call("rb_set_diag", ptr(H), M, M, ptr(rowsq), float(alpha), stream())
    if lam_rel is not None:
        lam = float(lam_rel) * float(H.diagonal().max().item())
    di = torch.empty(M, dtype=torch.float64, device=dev)
    call("rb_reginv_prepare", ptr(H), M, M, float(lam), ptr(di), stream())
    wb = _lib.lib().rb_cholesky_work_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=dev)
    call("rb_cholesky", ptr(H), M, M, ptr(work), wb, stream())
    return H, di, float(lam)


def normal_solve(J, K, H, di, r, lam, alpha=1.0, lo=None, refine=3, refine_tol=1e-14, info=None, return_y=False):
    """y = (alpha J J^T + lam I)^-1 r with the factor of normal_factor, then
    returns alpha J^T y (K-vector, FP64), or y itself with ``return_y``.

    The factor comes from tensor-core products, whose inputs are rounded
    (~1e-3 relative for TF32).  ``refine`` sweeps of FP64 iterative
    refinement make y the solution for the stored J itself: the residual
    r - alpha J (J^T y) - lam y takes FP64-accumulated GEMVs over J (two
    passes over J per sweep), and y += C^-1 residual with the factor C as the
    preconditioner, until ||residual|| <= refine_tol ||r||.  ``info`` (a dict)
    receives the sweeps done and the last relative residual."""
    op = J if isinstance(J, (StoredJacobian, SlabJacobian)) else StoredJacobian(J, K, lo)
    M = op.rows
    dev = H.device
    rr = torch.as_tensor(np.ascontiguousarray(r, dtype=np.float64), device=dev) if not torch.is_tensor(r) else r

    cwb = _lib.lib().rb_chol_solve_work_bytes(M)
    cwork = torch.empty(cwb, dtype=torch.uint8, device=dev)

    def precond(v):
        t = torch.empty(M, dtype=torch.float64, device=dev)
        call("rb_vec_mul", ptr(di), ptr(v), ptr(t), M, stream())
        call("rb_chol_solve", ptr(H), M, M, ptr(t), ptr(cwork), cwb, stream())
        out = torch.empty(M, dtype=torch.float64, device=dev)
        call("rb_vec_mul", ptr(di), ptr(t), ptr(out), M, stream())
        return out

    y = precond(rr)
    unchecked = True  # a solve whose result no finite residual norm vouches for
    sweeps, rel = 0, None
    u_now = None  # J^T y for the current y, when a residual pass left it
    if refine:
        rnorm = norm2(rr) or 1.0
        res = torch.empty(M, dtype=torch.float64, device=dev)
        for it in range(int(refine)):
            u, Ju = op.jt_then_j(y)
            res.copy_(rr)
            call("rb_axpby", M, -float(alpha), ptr(Ju), 1.0, ptr(res), stream())  # res = r - alpha J J^T y
            call("rb_axpby", M, -float(lam), ptr(y), 1.0, ptr(res), stream())  # res -= lam y
            rel = norm2(res) / rnorm
            unchecked = not np.isfinite(rel)
            if rel <= refine_tol:
                u_now = u
                break
            call("rb_axpby", M, 1.0, ptr(precond(res)), 1.0, ptr(y), stream())
            unchecked = True
            sweeps = it + 1
    if unchecked and not torch.cuda.is_current_stream_capturing():
        call("rb_chol_solve_status", stream())
    if info is not None:
        info.update(refine_sweeps=sweeps, refine_relres=rel, lam=float(lam))
    if return_y:
        return y
    if u_now is not None:  # the last residual pass already formed J^T y
        out = torch.empty_like(u_now)
        call("rb_axpby", u_now.numel(), float(alpha), ptr(u_now), 0.0, ptr(out), stream())
        return out
    return op.jt(y, alpha)


def reginv_under_device(J, K, r, lam, alpha=1.0, precision="tf32", lam_rel=None, refine=3, refine_tol=1e-14,
                        info=None, rowsq=None, Jb=None):
    """reginvunder (recon.py:429-509) for the rows of J (scaled by sqrt(alpha)):
    H = alpha J J^T + lam I on the tensor cores, unit-diagonal normalisation,
    FP64 Cholesky, FP64 refinement (normal_solve); returns alpha J^T y on the
    device (K-vector, FP64).  J is a stored matrix or a SlabJacobian."""
    if isinstance(J, SlabJacobian):  # J recomputed slab by slab on every pass
        H, di, lam = normal_factor_op(J, lam, alpha, precision, lam_rel, rowsq)
        return normal_solve(J, K, H, di, r, lam, alpha, None, refine, refine_tol, info)
    H, di, lo, lam = normal_factor(J, K, lam, alpha, precision, lam_rel, rowsq, Jb)
    return normal_solve(J, K, H, di, r, lam, alpha, lo, refine, refine_tol, info)


def gemv_t(J, K, y, alpha=1.0, beta=0.0, out=None, lo=None):
    """out = alpha J^T y + beta out on the device (J FP32 rows, y FP64); with
    ``lo`` the split remainder of J is added as well."""
    M, ldj = J.shape
    dev = J.device
    if out is None:
        out = torch.empty(K, dtype=torch.float64, device=dev)
    wb = _lib.lib().rb_gemv_t_work_bytes(K)
    work = torch.empty(wb, dtype=torch.uint8, device=dev)
    fn = "rb_gemv_t_bf16" if J.dtype == torch.bfloat16 else "rb_gemv_t"
    call(fn, ptr(J), M, K, ldj, ptr(y), float(alpha), float(beta), ptr(out), ptr(work), wb, stream())
    if lo is not None:  # J = hi + lo
        call("rb_gemv_t", ptr(lo), M, K, ldj, ptr(y), float(alpha), 1.0, ptr(out), ptr(work), wb, stream())
    return out
