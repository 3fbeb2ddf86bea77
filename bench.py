"""Benchmark: multi-RHS FEM forward solves on the 3M-tet box (RHS solves/s).

Workload (one "step" = one full forward pass, femrhs -> femlhs -> femsolve
-> femgetdet): box 100 x 100 x 50 mm at 1 mm Kuhn spacing (520,251 nodes,
3,000,000 tets), mua 0.01/mm, mus 1.0/mm, g 0, n 1.37, 64 sources on an 8x8
grid over x,y in [15,85] mm on z=0 and 64 detectors offset by 5 mm, CW.
All 128 columns are solved to the FP64 accuracy floor (mixed precision: FP32
block PCG inside FP64 refinement).  ``value`` = 128 RHS / device time per
step with inputs resident in HBM; ``e2e`` = the same through the public
``runforward`` API from host arrays (uploads and the phi/detval download
inside the timed region).  The working set (5 x 266 MB Krylov vectors) is
larger than L2, so no explicit flush is needed.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]
"""

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "RHS solves/s (3M tets, 64 src + 64 det, CW, <=1e-6 detector error)"
UNIT = "RHS/s"


def workload_cfg(spacing=1.0, omega=0.0):
    from redbirdpy_b200.meshgen import kuhn_box, grid_optodes

    node, elem = kuhn_box([100, 100, 50], spacing)
    return dict(node=node, elem=elem, prop=np.array([[0, 0, 1, 1], [0.01, 1.0, 0, 1.37]]),
                seg=np.ones(elem.shape[0], dtype=np.int32),
                srcpos=grid_optodes([15, 85], [15, 85], 8), srcdir=np.array([[0, 0, 1.0]]),
                detpos=grid_optodes([15, 85], [15, 85], 8, offset=(5, 5)), detdir=np.array([[0, 0, 1.0]]),
                omega=omega)


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_setup(n_gpus):
    import torch
    import torch.distributed as dist

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        torch.cuda.set_device(local)
        import datetime

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600),
                                device_id=torch.device("cuda", local))
    else:
        torch.cuda.set_device(0)
    return rank, world, local


def max_over_ranks(x, world):
    import torch
    import torch.distributed as dist

    if world == 1:
        return x
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(world):
    import torch.distributed as dist

    if world > 1:
        dist.barrier()


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return d.get("hbm_gbs", 6650.0), "measured"
    return 6650.0, "fallback"


def cpu_sample_port(cfg, ncol=1, maxiter=1000, tol=1e-10):
    """The oracle's port of the reference's femsolve(method='cg') on ncol
    columns of the same system (scipy CG per column, tol 1e-10, maxiter 1000:
    the reference defaults, solver.py:448-449, 717-754), one core.  The
    system comes from the oracle's femlhs / femrhs on the prepared mesh."""
    from oracle import femoracle as fo

    ocfg = {k: cfg[k] for k in ("node", "elem", "face", "area", "evol", "reff", "prop", "seg", "srcpos", "srcdir",
                                "detpos", "detdir", "omega")}
    A = fo.femlhs(ocfg, fo.deldotdel(ocfg["node"], ocfg["elem"], ocfg["evol"]))
    rhs, _, _, _ = fo.femrhs(dict(ocfg, srcpos=ocfg["srcpos"][:ncol], detpos=ocfg["detpos"][:1]))
    b = rhs[:, :ncol].toarray()
    from threadpoolctl import threadpool_limits

    with threadpool_limits(limits=1):  # one core, as reported
        t0 = time.perf_counter()
        fo.femsolve(A, b, method="cg", tol=tol, maxiter=maxiter)
        dt = time.perf_counter() - t0
    return ncol / dt, dt


def run_b200(args):
    import torch

    import redbirdpy_b200 as rbb
    from redbirdpy_b200 import engine

    rank, world, local = dist_setup(args.gpus)
    # meshprep of the 3M-tet box (reorientation, faces, areas, volumes, CSR
    # pattern and incidence on the device), after a small one that loads the
    # library and creates the context
    rbb.meshprep(workload_cfg(spacing=10.0))
    torch.cuda.synchronize()
    cfg = workload_cfg()
    t0 = time.perf_counter()
    cfg, sd = rbb.meshprep(cfg)
    mesh = engine.mesh_of(cfg)
    torch.cuda.synchronize()
    meshprep_s = time.perf_counter() - t0
    optics = engine.Optics.from_cfg(mesh, cfg)
    nrhs = cfg["srcpos"].shape[0] + cfg["detpos"].shape[0]

    def step(precision, profile=False, coarse="auto"):
        opt = engine.locate_optodes(mesh, cfg)
        B = opt.rhs(mesh)
        mat = engine.assemble(mesh, optics)
        X, info = engine.solve(mat, B, precision=precision, profile=profile, coarse=coarse)
        det = engine.getdet(mesh, opt, X)
        return det, X, info

    def timed(precision, k, w, profile=False, coarse="auto"):
        for _ in range(w):
            step(precision, coarse=coarse)
        torch.cuda.synchronize()
        barrier(world)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        infos = []
        for _ in range(k):
            det, X, info = step(precision, profile, coarse)
            infos.append(info)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / k
        barrier(world)
        return max_over_ranks(ms, world), det, infos

    clocks = ClockSampler(local)
    # mixed precision (the product form); clocks sampled during its timed region
    clocks.start()
    ms_mixed, det_mixed, infos = timed("mixed", args.steps, args.warmup)
    clk = clocks.stop()
    # per-kernel CUDA-event times of the Krylov loop (instrumented steps, not
    # part of the timed region above)
    _, _, pinfos = timed("mixed", 2, 0, profile=True)
    # plain FP64 form, same GPU, same accuracy target
    ms_fp64, det_fp64, infos64 = timed("fp64", max(1, min(args.steps, 3)), 1)
    # the same solve with the Jacobi preconditioner alone (no coarse space)
    ms_jac, _, infos_jac = timed("mixed", max(1, min(args.steps, 3)), 1, coarse=False)
    d64 = det_fp64.cpu().numpy()
    dmx = det_mixed.cpu().numpy()
    rel_err = float(np.max(np.abs(dmx - d64) / np.abs(d64)))

    # roofline of the SpMM kernel (dominant bytes per Krylov iteration)
    n, nnz, k = mesh.nn, mesh.nnz, nrhs
    # the product's own bytes: the CSR matrix (FP32 values, int32 indices) and
    # x and y once each, whatever plan the kernel walks
    spmm_bytes = nnz * (4 + 4) + 4 * (n + 1) + 2 * k * n * 4
    # r, q read + r written (FP32) (x += a p is in the p-update)
    upd_bytes = 3 * k * n * 4
    sp_ms = sum(i["spmm_ms"] for i in pinfos) / max(1, sum(i["spmm_launches"] for i in pinfos))
    up_ms = sum(i["update_ms"] for i in pinfos) / max(1, sum(i["update_launches"] for i in pinfos))
    peak, peak_kind = peaks()
    sp_gbs = spmm_bytes / (sp_ms * 1e-3) / 1e9 if sp_ms > 0 else None
    up_gbs = upd_bytes / (up_ms * 1e-3) / 1e9 if up_ms > 0 else None

    # assembly alone (femlhs kernel pair), CUDA events around 10 launches
    for _ in range(2):
        engine.assemble(mesh, optics)
    ea, eb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ea.record()
    for _ in range(10):
        engine.assemble(mesh, optics)
    eb.record()
    torch.cuda.synchronize()
    asm_ms = ea.elapsed_time(eb) / 10
    ne, nf = mesh.ne, mesh.nf
    pk = 8 if optics.kind == 0 else 8  # mua/musp per entity
    nprop = mesh.nn if optics.kind == 0 else ne
    # per tet: elem, deldotdel row, volume, its 4 incidence entries (+ their
    # 4 packed slot words with the contributor tables); per property entity
    # mua, musp and D; per nonzero: column index read, FP64 + FP32 value
    # written (+ the contributor mask); per node: the three row pointers and
    # the FP64 + FP32 reciprocal diagonal; per boundary face: nodes and area
    tab = mesh.inc_slot is not None
    asm_bytes = (ne * (16 + 80 + 8 + 16 + (16 if tab else 0)) + nprop * (2 * pk + 8)
                 + nnz * (4 + 8 + 4 + (4 if tab else 0)) + n * (4 * 3 + 12) + nf * (12 + 8 + 12))
    asm_gbs = asm_bytes / (asm_ms * 1e-3) / 1e9

    # end to end through the public API (host arrays in, numpy out)
    host_cfg = cfg
    # warm-up: two results held at once, the steady state of a loop that
    # keeps the previous phi while the next call runs (fills the pinned pool)
    warm = [rbb.runforward(host_cfg) for _ in range(2)]
    del warm
    torch.cuda.synchronize()
    barrier(world)
    t0 = time.perf_counter()
    ke = max(1, min(args.steps, 3))
    for _ in range(ke):
        det_h, phi_h = rbb.runforward(host_cfg)
    torch.cuda.synchronize()
    e2e_s = max_over_ranks((time.perf_counter() - t0) / ke, world)
    # what one runforward call uploads: the optode positions (located on the
    # device every call), the per-tet labels (int32) and the label property
    # table (mua, musp, g rows) expanded per tet on the device; the mesh is
    # uploaded once and kept on the device across calls (as redbirdpy keeps
    # the prepared mesh in cfg)
    props = np.atleast_2d(cfg["prop"])
    h2d = int(cfg["srcpos"].size * 8 + cfg["detpos"].size * 8 + np.size(cfg["seg"]) * 4
              + props.shape[0] * min(3, props.shape[1]) * 8)
    d2h = det_h.nbytes + phi_h.nbytes

    # DRAM bytes per launch from an earlier ncu capture of this workload,
    # stored beside the summaries (not measured in this run)
    traffic = {}
    tp = os.path.join(ROOT, "profiles", "traffic_per_launch.json")
    if os.path.exists(tp):
        traffic = json.load(open(tp))
    it = infos[-1]
    spk = it.get("spmm_kernel", "spmm_pair_kernel")
    spmm_desc = {"vc_spmm_kernel": "vc_spmm_kernel (FP32 SpMM of the scaled matrix over 2x2x2 spatial row groups, one gather "
                                   "per group column, 128 RHS, fused p.Ap)",
                 "spmm_blk_kernel": "spmm_blk_kernel (FP32 CSR SpMM over 2x2x2 spatial row groups, one gather per "
                                    "group column, 128 RHS, fused p.Ap)",
                 "spmm_pair_kernel": "spmm_pair_kernel (FP32 CSR SpMM, two rows per warp over their column union, "
                                     "128 RHS, fused p.Ap)"}[spk]
    asm_kernel = "femlhs_tab_kernel" if mesh.inc_slot is not None else "femlhs_rows_kernel"
    out = {
        "metric": METRIC, "value": round(world * nrhs / (ms_mixed * 1e-3), 3), "unit": UNIT,
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_mixed, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
        "data": "synthetic",
        "config": {"workload": "box 100x100x50 mm, 1 mm Kuhn (520251 nodes, 3000000 tets), 64 src + 64 det, CW",
                   "nnz": nnz, "nrhs": nrhs,
                   "precision": "mixed (FP32 PCG in FP64 refinement; three-level V-cycle)",
                   "l2": "working set > L2 (5 x 266 MB vectors), no flush", "parallelism": f"replicas x{world}"},
        "fp64_value": round(world * nrhs / (ms_fp64 * 1e-3), 3), "fp64_ms_per_step": round(ms_fp64, 3),
        "mixed_speedup_vs_fp64": round(ms_fp64 / ms_mixed, 3),
        "det_max_rel_err_vs_fp64": rel_err,
        "krylov": {"iters": it["iters"], "sweeps": it["outer"], "relres": it["relres"], "flag": it["flag"],
                   "fp64_iters": infos64[-1]["iters"], "coarse_aggregates": it["coarse_nc"],
                   "coarse_ms_per_iter": round(sum(i["coarse_ms"] for i in pinfos)
                                               / max(1, sum(i["coarse_launches"] for i in pinfos)), 4),
                   "jacobi_only_ms_per_step": round(ms_jac, 3), "jacobi_only_iters": infos_jac[-1]["iters"]},
        "gpu_launches": int(sum(i["launches"] for i in infos) / len(infos)) + 6,
        "roofline": {"bound": "hbm", "kernel": spmm_desc,
                     "achieved": round(sp_gbs, 1) if sp_gbs else None, "peak": peak, "unit": "GB/s",
                     "frac": round(sp_gbs / peak, 4) if sp_gbs else None, "peak_source": peak_kind,
                     "algorithmic_bytes": spmm_bytes, "launch_ms": round(sp_ms, 4),
                     "traffic": traffic.get(spk + "<EPI_PQDOT>"),
                     "traffic_source": "stored: an earlier ncu capture of this workload, not measured in this run"},
        "roofline_update": {"kernel": "vc_update_kernel<float> (r update + r.r)",
                            "achieved": round(up_gbs, 1) if up_gbs else None,
                            "unit": "GB/s", "frac": round(up_gbs / peak, 4) if up_gbs else None,
                            "algorithmic_bytes": upd_bytes, "launch_ms": round(up_ms, 4),
                            "traffic": traffic.get("vc_update_kernel<float,32,1>"),
                            "traffic_source": "stored (earlier ncu capture)"},
        "roofline_assembly": {"kernel": asm_kernel + " (+ dcoeff prologue)", "achieved": round(asm_gbs, 1),
                              "unit": "GB/s", "frac": round(asm_gbs / peak, 4), "algorithmic_bytes": asm_bytes,
                              "launch_ms": round(asm_ms, 4), "traffic": traffic.get(asm_kernel + "<real,per-tet>"),
                              "traffic_source": "stored (earlier ncu capture)"},
        "e2e": {"value": round(world * nrhs / e2e_s, 3), "unit": UNIT, "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": int(d2h)},
        "clocks": clk,
        "meshprep": {"seconds": round(meshprep_s, 3),
                     "what": "rbb.meshprep + device mesh (reorientation, boundary faces, areas, tet and node "
                             "volumes, incidence, CSR pattern, assembly tables) of the 3M-tet box, host arrays in",
                     "reference_seconds": 95, "reference_source": "the survey's probe of redbirdpy's meshprep "
                                                                  "(numpy fallbacks, _femnz loop) at this size"},
    }
    # each section starts with torch's cached device memory released: the GN
    # section leaves tens of GB of Jacobian blocks in the allocator's cache
    if not args.no_gn:
        torch.cuda.empty_cache()
        out["gn"] = run_gn_step(cfg, mesh, world, args)
    if not args.no_adjoint:
        torch.cuda.empty_cache()
        out["adjoint"] = run_adjoint(world, args)
    if not args.no_batch:
        torch.cuda.empty_cache()
        out["batch"] = run_batch(world, args)
    if rank == 0 and world == 1 and not args.no_cpu:
        v, dt = cpu_sample_port(cfg, ncol=1)
        out["cpu_baseline"] = {"value": round(v, 5), "unit": UNIT, "cores": 1, "kind": "port",
                               "sample": f"1 of 128 columns, oracle port of femsolve(method='cg') "
                                         f"tol 1e-10 maxiter 1000 (scipy CG), {dt:.1f} s"}
    if rank == 0:
        print(json.dumps(out))
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


def gn_truth(node):
    """Two spherical inclusions (r = 8 mm): mua 0.025 at (35,50,20), mus 2.0 at (65,50,25)."""
    nn = node.shape[0]
    prop = np.column_stack([np.full(nn, 0.01), np.full(nn, 1.0), np.zeros(nn), np.full(nn, 1.37)])
    prop[np.linalg.norm(node - [35.0, 50.0, 20.0], axis=1) < 8.0, 0] = 0.025
    prop[np.linalg.norm(node - [65.0, 50.0, 25.0], axis=1) < 8.0, 1] = 2.0
    return prop


def tiles_flop(mesh, M=8192):
    """Algorithmic flop of J J^T over the 256 x 256 tiles on or above the diagonal."""
    nbt = (M + 255) // 256
    return nbt * (nbt + 1) // 2 * 256 * 256 * (2 * mesh.nn) * 2


def run_gn_step(cfg, mesh, world, args):
    """One Gauss-Newton iteration of the 3M-tet frequency-domain problem
    (64 x 64 complex data -> 8192 real rows, node-wise mua and D -> 1,040,502
    columns): forward (mixed COCG) -> exact adjoint Jacobian rows (FP32) ->
    Frobenius scaling -> J J^T on the tensor cores (TF32) -> FP64 Cholesky ->
    J^T y.  Beside it the plain FP64 form on the same GPU: FP64 COCG,
    FP64 Jacobian, FP64 J J^T (cuBLAS DGEMM through torch, the library
    baseline), the same FP64 Cholesky."""
    import torch

    from redbirdpy_b200 import engine
    from redbirdpy_b200.forward import forward_device

    gcfg = dict(cfg)
    gcfg["omega"] = 2 * np.pi * 1e8
    gcfg["prop"] = gn_truth(cfg["node"])
    gcfg.pop("seg", None)
    det_t, _, _, _, _ = forward_device(gcfg)
    rng = np.random.default_rng(1)
    d = det_t.cpu().numpy().ravel()
    data = d * (1 + 0.01 * rng.standard_normal(d.shape)) * np.exp(1j * np.deg2rad(0.5) * rng.standard_normal(d.shape))
    bg = gn_truth(cfg["node"])
    bg[:, 0], bg[:, 1] = 0.01, 1.0
    gcfg["prop"] = bg
    sd = np.column_stack([np.meshgrid(np.arange(64), 64 + np.arange(64))[0].ravel(),
                          np.meshgrid(np.arange(64), 64 + np.arange(64))[1].ravel(), np.ones(4096)])
    stages = {}

    def timed_stage(name, fn):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        r = fn()
        e1.record()
        torch.cuda.synchronize()
        stages[name] = stages.get(name, 0.0) + e0.elapsed_time(e1)
        return r

    def apply_update(prop, dmu):
        """runrecon's update (mua, and D through musp: D = 1/(3(mua+musp)))."""
        nn = prop.shape[0]
        d_old = 1.0 / (3.0 * (prop[:, 0] + prop[:, 1]))
        prop[:, 0] += dmu[:nn]
        prop[:, 1] = 1.0 / (3.0 * (d_old + dmu[nn:2 * nn])) - prop[:, 0]

    state = {"phi": None}
    refine = 3  # FP64 refinement sweeps of the normal equations (at most)

    def step_mixed(jdtype=torch.float32, apply=True, gram_prec="bf16"):
        # one iteration of the GN loop: the forward solve starts from the
        # previous iterate's fields, and the update is applied at the end
        det, phi, _, _, _ = timed_stage("forward", lambda: forward_device(gcfg, x0=state["phi"]))
        J, K = timed_stage("jacobian", lambda: engine.jacobian_matrix(mesh, phi, sd, ("mua", "D"), "exact",
                                                                      dtype=jdtype,
                                                                      acc64=jdtype == torch.float32))
        y = det.cpu().numpy().ravel()
        mis = data - y
        mis = np.concatenate([mis.real, mis.imag])
        # row sums of squares: the Frobenius scale and the exact diagonal of
        # J J^T (the product's own diagonal carries the TF32 input rounding,
        # which lam = 0.05 max(diag) would inherit)
        bfc = gram_prec == "bf16" and J.dtype == torch.float32
        sums = timed_stage("sumsq", lambda: engine.row_sumsq(J, K, bf16_copy=bfc))
        rowsq, tot = sums[0], sums[1]
        s2 = 1.0 / float(tot.item())
        # tf32x3 leaves J as its TF32 part and returns the remainder: the
        # refinement below runs over both, i.e. over the FP32 rows; 'bf16'
        # forms the product from the BF16 copy made in the same pass as the
        # row sums and refines over the FP32 rows
        H, lo = timed_stage("gram", lambda: engine.gram(sums[2] if bfc else J, K, s2, gram_prec))
        del sums
        engine.call("rb_set_diag", engine.ptr(H), H.shape[0], H.shape[0], engine.ptr(rowsq), s2, engine.stream())
        lam = 0.05 * float(H.diagonal().max().item())
        M = J.shape[0]
        di = torch.empty(M, dtype=torch.float64, device=J.device)

        def chol():
            engine.call("rb_reginv_prepare", engine.ptr(H), M, M, lam, engine.ptr(di), engine.stream())
            wb = engine._lib.lib().rb_cholesky_work_bytes()
            work = torch.empty(wb, dtype=torch.uint8, device=J.device)
            engine.call("rb_cholesky", engine.ptr(H), M, M, engine.ptr(work), wb, engine.stream())

        timed_stage("cholesky", chol)
        # solve with FP64 refinement over the stored J, then J^T y
        rinfo = {}
        dmu = timed_stage("solve_refine_jty", lambda: engine.normal_solve(
            J, K, H, di, mis, lam, s2, lo, refine=refine, info=rinfo).cpu().numpy())
        state["refine"] = rinfo
        state["det"] = det
        del J, H, lo
        if apply:
            apply_update(gcfg["prop"], dmu)
            state["phi"] = phi
        return dmu

    # warm-up (GN iteration 1, from zero fields), then timed iterations 2..
    # (device time, CUDA events around each stage); the state before the last
    # timed iteration is kept for the FP64 form
    step_mixed()
    torch.cuda.synchronize()
    stages.clear()
    ks = max(1, min(args.steps, 2))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    # clocks during the timed GN iterations: the tensor-core product runs at
    # the 1 kW power cap, where the SM clock settles well below its maximum
    gclk = ClockSampler(torch.cuda.current_device())
    gclk.start()
    e0.record()
    for i in range(ks):
        if i == ks - 1:
            snap = (gcfg["prop"].copy(), state["phi"])
        dmu_mixed = step_mixed()
    e1.record()
    torch.cuda.synchronize()
    gn_clocks = gclk.stop()
    ms = max_over_ranks(e0.elapsed_time(e1) / ks, world)
    mixed_stages = {k: round(v / ks, 2) for k, v in stages.items()}

    # plain FP64 form of the same GN iteration (same state, same warm start)
    def step_fp64():
        gcfg["prop"] = snap[0].copy()
        det, phi, _, _, _ = forward_device(gcfg, precision="fp64", x0=snap[1])
        state["det64"] = det.cpu().numpy()
        cols, det0, ndet, psrc, pdet, _, _ = engine.pair_map(sd)
        nn = mesh.nn
        K = 2 * nn
        M = 2 * len(psrc)
        J = torch.zeros((M, K), dtype=torch.float64, device=phi.device)
        colsd, ps, pd = engine._i32(cols, phi.device), engine._i32(psrc, phi.device), engine._i32(pdet, phi.device)
        for p, w in enumerate((engine._lib.RB_JAC_MUA_NODAL, engine._lib.RB_JAC_D)):
            engine.call("rb_jac", engine.ctypes.byref(mesh.struct), w, engine.ptr(phi), engine._lib.RB_C128,
                        phi.shape[1], engine.ptr(colsd), len(cols), det0, ndet, engine.ptr(ps), engine.ptr(pd),
                        len(psrc), engine.ptr(J[:, p * nn:]), K, engine._lib.RB_JAC_SPLIT_F64, mesh.rmax, mesh.emax,
                        engine.ptr(mesh.evol), engine.ptr(mesh.ddd if p else None), engine.stream())
        y = det.cpu().numpy().ravel()
        mis = data - y
        mis = np.concatenate([mis.real, mis.imag])
        s2 = 1.0 / float(torch.linalg.vector_norm(J).item()) ** 2
        H = torch.matmul(J, J.T) * s2
        lam = 0.05 * float(H.diagonal().max().item())
        di = torch.empty(M, dtype=torch.float64, device=J.device)
        engine.call("rb_reginv_prepare", engine.ptr(H), M, M, lam, engine.ptr(di), engine.stream())
        wb = engine._lib.lib().rb_cholesky_work_bytes()
        work = torch.empty(wb, dtype=torch.uint8, device=J.device)
        engine.call("rb_cholesky", engine.ptr(H), M, M, engine.ptr(work), wb, engine.stream())
        t = di * torch.as_tensor(mis, device=J.device)
        cwb = engine._lib.lib().rb_chol_solve_work_bytes(M)
        cwork = torch.empty(cwb, dtype=torch.uint8, device=J.device)
        engine.call("rb_chol_solve", engine.ptr(H), M, M, engine.ptr(t), engine.ptr(cwork), cwb, engine.stream())
        dmu = torch.mv(J.T, di * t) * s2
        return dmu.cpu().numpy()

    refine_info = dict(state.get("refine", {}))
    det_mixed = state["det"].cpu().numpy()
    ms64 = None
    err = None
    det_err = None
    if not args.no_fp64_gn:
        torch.cuda.synchronize()
        f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f0.record()
        dmu64 = step_fp64()
        f1.record()
        torch.cuda.synchronize()
        ms64 = max_over_ranks(f0.elapsed_time(f1), world)
        err = float(np.linalg.norm(dmu_mixed - dmu64) / np.linalg.norm(dmu64))
        det_err = float(np.max(np.abs(det_mixed - state["det64"]) / np.abs(state["det64"])))
    M, K = 8192, 2 * mesh.nn
    nbt = (M + 255) // 256
    tiles = nbt * (nbt + 1) // 2  # 256 x 256 tiles on or above the diagonal
    gram_flop = tiles * 256 * 256 * K * 2
    gram_ms = mixed_stages.get("gram")
    # the same iteration with the product in TF32 (kind::tf32 on the FP32
    # rows themselves), same state as the FP64 comparison
    tf32 = None
    if not args.no_fp64_gn:
        gcfg["prop"] = snap[0].copy()
        state["phi"] = snap[1]
        step_mixed(apply=False, gram_prec="tf32")  # first call of the TF32 kernels
        torch.cuda.synchronize()
        stages.clear()
        b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        b0.record()
        dmu_t = step_mixed(apply=False, gram_prec="tf32")
        b1.record()
        torch.cuda.synchronize()
        tms = max_over_ranks(b0.elapsed_time(b1), world)
        tf32 = {"ms_per_iter": round(tms, 1), "breakdown_ms": {k: round(v, 2) for k, v in stages.items()},
                "speedup_vs_fp64": round(ms64 / tms, 3), "iters_per_s": round(1e3 / tms, 4) * world,
                "dmu_rel_err_vs_fp64": float(np.linalg.norm(dmu_t - dmu64) / np.linalg.norm(dmu64)),
                "gram_tflops": round(tiles_flop(mesh) / (stages["gram"] * 1e-3) / 1e12, 1),
                "refinement": dict(state.get("refine", {})),
                "note": "J J^T on the FP32 rows in TF32 (kind::tf32); the FP64 refinement runs over the same rows"}
    # the same iteration with the Jacobian never stored: node slabs of a
    # quarter of the mesh recomputed on every pass (the mode a mesh whose J
    # exceeds HBM takes), same state as the FP64 comparison
    slab = None
    if not args.no_fp64_gn:
        gcfg["prop"] = snap[0].copy()

        def step_slab(width):
            det, phi, _, _, _ = forward_device(gcfg, x0=snap[1])
            op = engine.SlabJacobian(mesh, phi, sd, ("mua", "D"), "exact", width, acc64=True)
            y = det.cpu().numpy().ravel()
            mis = data - y
            mis = np.concatenate([mis.real, mis.imag])
            rowsq, tot = op.row_sumsq()
            s2 = 1.0 / float(tot.item())
            H, di, lam = engine.normal_factor_op(op, 0.0, s2, "bf16", lam_rel=0.05, rowsq=rowsq)
            rinfo = {}
            dmu = engine.normal_solve(op, op.K, H, di, mis, lam, s2, None, refine=refine, info=rinfo)
            return dmu.cpu().numpy(), op.passes, rinfo

        width = (mesh.nn + 3) // 4
        step_slab(width)
        torch.cuda.synchronize()
        b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        b0.record()
        dmu_s, passes, rinfo_s = step_slab(width)
        b1.record()
        torch.cuda.synchronize()
        sms = max_over_ranks(b0.elapsed_time(b1), world)
        slab = {"ms_per_iter": round(sms, 1), "slab_nodes": width, "jacobian_passes": passes,
                "jacobian_slab_bytes": int(8192 * 2 * width * 4),
                "jacobian_stored_bytes": int(8192 * 2 * mesh.nn * 4),
                "refine_sweeps": rinfo_s.get("refine_sweeps"),
                "dmu_rel_err_vs_fp64": float(np.linalg.norm(dmu_s - dmu64) / np.linalg.norm(dmu64))}
    tflops = gram_flop / (gram_ms * 1e-3) / 1e12 if gram_ms else None
    pk, pk_src, pk_sus = 1590.0, "fallback bf16 (burst), no MEASURED_PEAKS.json", 1400.0
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        mp = json.load(open(p))
        v = mp.get("bf16_tflops")
        if v:
            pk, pk_src = float(v), "measured bf16 (burst)"
        pk_sus = float(mp.get("bf16_tflops_sustained") or pk_sus)
    return {
        "workload": f"{mesh.ne} tets / {mesh.nn} nodes, omega=2*pi*100MHz, 64x64 complex pairs -> 8192 real rows, "
                    f"mua+D nodal (K={2 * mesh.nn}), FP32 Jacobian rows (products formed in FP64), J J^T on the tensor cores from their BF16 "
                    f"copy (made in the row-sum pass) + FP64 refinement of the normal equations over the FP32 rows; "
                    f"lam = 0.05 max diag(J J^T) from the exact row sums; GN iterations 2..{ks + 1} of the loop "
                    f"(forward warm-started from the previous iterate's fields), iteration 1 untimed",
        "iters_per_s": round(1e3 / ms, 4) * world, "ms_per_iter": round(ms, 1), "breakdown_ms": mixed_stages,
        "fp64_iters_per_s": round(1e3 / ms64, 4) * world if ms64 else None,
        "fp64_ms_per_iter": round(ms64, 1) if ms64 else None,
        "speedup_vs_fp64": round(ms64 / ms, 3) if ms64 else None,
        "dmu_rel_err_vs_fp64": err,
        "forward_det_max_rel_err_vs_fp64": det_err,
        "refinement": refine_info,
        "roofline_gram": {"bound": "tensor", "kernel": "gram_tf32_kernel<true> (tcgen05 kind::f16, BF16 A and B, "
                                                       "FP32 accumulation drained to FP64, 256x256 tiles)",
                          "achieved": round(tflops, 1) if tflops else None, "unit": "TFLOP/s",
                          "algorithmic_flop": gram_flop, "peak": pk, "peak_source": pk_src,
                          "frac": round(tflops / pk, 4) if (tflops and pk) else None,
                          "sustained_peak": pk_sus,
                          "frac_of_sustained": round(tflops / pk_sus, 4) if (tflops and pk_sus) else None,
                          "note": "the GN step runs at the 1 kW power cap (sw_power_cap), where the clocks reach "
                                  "the sustained figure"},
        "clocks": gn_clocks,
        "tf32_form": tf32,
        "slab_recompute_form": slab,
    }


def run_profile(args):
    """A short, fixed workload for ncu captures (``--profile-run``): the
    forward step ``--warmup + --steps`` times on the box meshed at
    ``--spacing`` mm, then (``--with-gn``) one mixed-precision GN iteration
    of the frequency-domain problem on the same mesh."""
    import torch

    import redbirdpy_b200 as rbb
    from redbirdpy_b200 import engine

    torch.cuda.set_device(0)
    cfg = workload_cfg(spacing=args.spacing)
    cfg, sd = rbb.meshprep(cfg)
    mesh = engine.mesh_of(cfg)
    optics = engine.Optics.from_cfg(mesh, cfg)
    for _ in range(args.warmup + args.steps):
        opt = engine.locate_optodes(mesh, cfg)
        B = opt.rhs(mesh)
        mat = engine.assemble(mesh, optics)
        X, info = engine.solve(mat, B)
        det = engine.getdet(mesh, opt, X)
    torch.cuda.synchronize()
    out = {"profile_run": True, "nn": mesh.nn, "ne": mesh.ne, "iters": info["iters"]}
    if args.with_gn:
        class A:  # one timed GN iteration, no FP64 comparison
            steps, no_fp64_gn = 1, True
        out["gn"] = run_gn_step(cfg, mesh, 1, A)
    print(json.dumps(out))


def _masked_log_amp_loss(own, tgt):
    """0.5 sum (log|det| - log|target|)^2 over every instance's own (detector,
    source) pairs of the stacked batch matrix, as one set of tensor ops."""
    import torch

    def loss(det):
        d = torch.where(own, det, torch.ones_like(det))
        t = torch.where(own, tgt, torch.ones_like(tgt))
        return 0.5 * torch.sum((torch.log(torch.abs(d)) - torch.log(torch.abs(t))) ** 2)
    return loss


def _log_amp_loss(parts, targets):
    import torch

    return sum(0.5 * torch.sum((torch.log(torch.abs(p)) - torch.log(torch.abs(t))) ** 2)
               for p, t in zip(parts, targets))


def run_adjoint(world, args):
    """Adjoint gradient and Jacobian rows on the 375k-tet box (51 x 51 x 26
    nodes at 2 mm), per-node mua ~ U[0.008, 0.012], mus ~ U[0.9, 1.1]
    (seed 0), 32 sources (8 x 4 grid) and 32 detectors (offset 5 mm) on z = 0,
    CW.  One step = forward + autograd backward of
    0.5 ||log|det| - log|target|||^2 (target: +10% mua) through the
    hand-written adjoint; beside it the full FP32 Jmua and JD rows
    (1024 x 67,626 each) and their HBM write rate."""
    import torch

    import redbirdpy_b200 as rbb
    from redbirdpy_b200 import engine
    from redbirdpy_b200.adjoint import DeviceModel, detector_values
    from redbirdpy_b200.meshgen import kuhn_box

    node, elem = kuhn_box([100, 100, 50], 2.0)
    nn = node.shape[0]
    rng = np.random.default_rng(0)
    prop = np.column_stack([rng.uniform(0.008, 0.012, nn), rng.uniform(0.9, 1.1, nn), np.zeros(nn),
                            np.full(nn, 1.37)])
    src = np.column_stack([np.repeat(np.linspace(15, 85, 8), 4), np.tile(np.linspace(30, 70, 4), 8), np.zeros(32)])
    cfg = dict(node=node, elem=elem, prop=prop, srcpos=src, srcdir=np.array([[0, 0, 1.0]]), detpos=src + [5, 5, 0],
               detdir=np.array([[0, 0, 1.0]]), omega=0.0)
    cfg, sd = rbb.meshprep(cfg)
    out = {"workload": f"{elem.shape[0]} tets / {nn} nodes, 32 src x 32 det, CW, per-node mua and D"}
    mua0 = torch.as_tensor(prop[:, 0].copy(), device="cuda")
    d0 = torch.as_tensor(1.0 / (3.0 * (prop[:, 0] + prop[:, 1])), device="cuda")
    grads = {}
    for prec in ("mixed", "fp64"):
        model = DeviceModel(cfg, precision=prec)
        with torch.no_grad():
            target = detector_values(model, mua0 * 1.1, d0)

        def step():
            mua = mua0.clone().requires_grad_(True)
            dco = d0.clone().requires_grad_(True)
            loss = _log_amp_loss([detector_values(model, mua, dco)], [target])
            loss.backward()
            return mua.grad, dco.grad

        for _ in range(2):
            step()
        torch.cuda.synchronize()
        # each step timed on its own; the median is reported (a step of a
        # shared machine now and then takes several times longer)
        ks = max(3, min(args.steps, 5))
        times = []
        for _ in range(ks):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            gm, gd = step()
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        ms = max_over_ranks(float(np.median(times)), world)
        grads[prec] = (gm, gd)
        out[f"{prec}_ms_per_gradient"] = round(ms, 2)
        out[f"{prec}_ms_steps"] = [round(t, 2) for t in times]
    gm, gd = grads["mixed"]
    rm, rd = grads["fp64"]
    out["grad_rel_err_vs_fp64"] = float(max((torch.abs(gm - rm).max() / torch.abs(rm).max()).item(),
                                            (torch.abs(gd - rd).max() / torch.abs(rd).max()).item()))
    out["gradients_per_s"] = round(world * 1e3 / out["mixed_ms_per_gradient"], 3)
    # full FP32 Jacobian rows (mua and D), as the GN step builds them
    model = DeviceModel(cfg)
    phi, _ = model.fields(mua0, d0)
    mesh = model.mesh
    ns = model.opt.nsrc
    sdj = np.column_stack([np.tile(np.arange(ns), ns), ns + np.repeat(np.arange(ns), ns), np.ones(ns * ns)])
    for _ in range(2):
        J, K = engine.jacobian_matrix(mesh, phi, sdj, ("mua", "D"), "exact")
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(3):
        J, K = engine.jacobian_matrix(mesh, phi, sdj, ("mua", "D"), "exact")
    e1.record()
    torch.cuda.synchronize()
    jms = e0.elapsed_time(e1) / 3
    jbytes = J.shape[0] * K * 4
    peak, _ = peaks()
    out["jacobian"] = {"rows": int(J.shape[0]), "cols": int(K), "ms": round(jms, 3),
                       "write_gbs": round(jbytes / (jms * 1e-3) / 1e9, 1),
                       "frac_of_hbm": round(jbytes / (jms * 1e-3) / 1e9 / peak, 4),
                       "note": "both quantities (rb_jac_multi: mua_nodal, D) and the clear of the row padding"}
    return out


def engine_status(code):
    from redbirdpy_b200.engine import INSTANCE_STATUS

    return INSTANCE_STATUS[int(code)]


def run_batch(world, args):
    """256 uneven box instances (seed 2; extents ~ U[30, 80] mm per axis,
    spacing in {2, 3, 4} mm, per-node mua ~ U[0.005, 0.03], mus ~ U[0.5, 2],
    4-16 top-surface sources and 4-16 detectors each, CW): forward + adjoint
    gradient of a log-amplitude misfit (target: +10% mua) for all instances
    as one block-diagonal system (one assembly, one mixed-precision solve,
    one adjoint contraction), against a loop over the instances' own models
    (timed on the first 32)."""
    import torch

    import redbirdpy_b200 as rbb
    from redbirdpy_b200 import engine
    from redbirdpy_b200.adjoint import BatchModel, DeviceModel, detector_values
    from redbirdpy_b200.meshgen import batch_boxes

    cfgs = [rbb.meshprep(c)[0] for c in batch_boxes(256, seed=2)]
    nn = sum(c["node"].shape[0] for c in cfgs)
    ne = sum(c["elem"].shape[0] for c in cfgs)
    bm = BatchModel(cfgs)
    mua0 = torch.as_tensor(np.concatenate([c["prop"][:, 0] for c in cfgs]), device="cuda")
    d0 = torch.as_tensor(np.concatenate([1.0 / (3.0 * (c["prop"][:, 0] + c["prop"][:, 1])) for c in cfgs]),
                         device="cuda")
    # launch shapes of the solve from the autotuner (one-time, untimed)
    tuned = dict(bm.tune(mua0, d0))
    bm_mat = engine.assemble(bm.mesh, bm.optics(mua0, d0))
    key = engine.solve_tuner.bucket(bm_mat, bm.B.shape[1], bm.solve_kw)
    tune_ms = {f"lanes={a},check_every={b}": round(v, 2) for (a, b), v in engine.solve_tuner.timings[key].items()}
    del bm_mat
    with torch.no_grad():
        tgt_all = detector_values(bm, mua0 * 1.1, d0)
        targets = bm.split(tgt_all)
    loss_fn = _masked_log_amp_loss(bm.own, tgt_all)

    def step():
        mua = mua0.clone().requires_grad_(True)
        dco = d0.clone().requires_grad_(True)
        loss_fn(detector_values(bm, mua, dco)).backward()
        return mua.grad

    for _ in range(2):
        step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ks = max(1, min(args.steps, 3))
    e0.record()
    for _ in range(ks):
        g = step()
    e1.record()
    torch.cuda.synchronize()
    ms = max_over_ranks(e0.elapsed_time(e1) / ks, world)
    # the same step replayed from one CUDA graph (fixed solve budget from a
    # checked calibration solve; no host round trips inside the step)
    from redbirdpy_b200.adjoint import CapturedStep

    cap = CapturedStep(bm, loss_fn, mua0, d0)
    for _ in range(3):
        cap(mua0, d0)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(ks):
        cap(mua0, d0)
    e1.record()
    torch.cuda.synchronize()
    ms_graph = max_over_ranks(e0.elapsed_time(e1) / ks, world)
    graph_status = cap.status.cpu().numpy()
    g_graph = cap.gmua.clone()
    cap.release()
    g_err = float((torch.abs(g_graph - g).max() / torch.abs(g).max()).item())
    # accuracy: detector values against the FP64 form of the same batch
    with torch.no_grad():
        dm = detector_values(bm, mua0, d0)
        d64 = detector_values(BatchModel(cfgs, precision="fp64"), mua0, d0)
    # each instance's own (detector, source) pairs; the rest of the
    # block-diagonal columns are other instances' sources
    err = max(float((torch.abs(a - b) / torch.abs(b)).max().item())
              for a, b in zip(bm.split(dm), bm.split(d64)) if b.numel())
    # loop over per-instance models (first 32 instances)
    nloop = 32
    models = [DeviceModel(c) for c in cfgs[:nloop]]
    tl = []
    for i, m in enumerate(models):
        mu0 = mua0[bm.node_off[i]:bm.node_off[i + 1]]
        dd0 = d0[bm.node_off[i]:bm.node_off[i + 1]]
        mu = mu0.clone().requires_grad_(True)
        dc = dd0.clone().requires_grad_(True)
        _log_amp_loss([detector_values(m, mu, dc)], [targets[i]]).backward()  # warm-up
    torch.cuda.synchronize()
    l0, l1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    l0.record()
    for i, m in enumerate(models):
        mu = mua0[bm.node_off[i]:bm.node_off[i + 1]].clone().requires_grad_(True)
        dc = d0[bm.node_off[i]:bm.node_off[i + 1]].clone().requires_grad_(True)
        _log_amp_loss([detector_values(m, mu, dc)], [targets[i]]).backward()
    l1.record()
    torch.cuda.synchronize()
    loop_ms = l0.elapsed_time(l1) / nloop
    st = np.asarray(bm.status)
    return {"workload": f"256 instances, {nn} nodes / {ne} tets in total, {bm.S} source + {bm.D} detector columns",
            "convergence": "per (instance, column): ||b_i - A_i x_i|| / ||b_i|| <= tol for each instance",
            "autotuned": {"chosen": {k: tuned[k] for k in ("spmm_lanes", "check_every")},
                          "solve_ms_per_candidate": tune_ms,
                          "note": "spmm_lanes 0 = the layout chosen from the column count"},
            "inst_relres_max": float(np.max(bm.relres)),
            "inst_status": {engine_status(k): int(np.sum(st == k)) for k in np.unique(st)},
            "instances_per_s": round(world * 256 / (ms * 1e-3), 2), "ms_per_batch": round(ms, 2),
            "graph": {"instances_per_s": round(world * 256 / (ms_graph * 1e-3), 2),
                      "ms_per_batch": round(ms_graph, 2), "budget": list(cap.budget),
                      "instances_converged": int(np.sum(graph_status == 0)),
                      "grad_rel_err_vs_checked": g_err},
            "loop_instances_per_s": round(world * 1e3 / loop_ms, 2),
            "loop_sample": f"first {nloop} instances, one model each (same kernels, launch-bound)",
            "speedup_vs_loop": round(loop_ms * 256 / ms, 2), "det_max_rel_err_vs_fp64": err}


_REF = {}


def _ref_init():
    from threadpoolctl import threadpool_limits

    _REF["limits"] = threadpool_limits(limits=1)


def _ref_worker(args):
    """One column of the reference's femsolve(method='cg') in a pool worker
    (one BLAS thread per worker, the system loaded once per worker)."""
    path, col, tol, maxiter = args
    import numpy as np
    from scipy import sparse
    from scipy.sparse.linalg import cg

    if _REF.get("path") != path:
        z = np.load(path)
        _REF["A"] = sparse.csr_matrix((z["data"], z["indices"], z["indptr"]))
        _REF["R"] = sparse.csc_matrix((z["rdata"], z["rindices"], z["rindptr"]), shape=tuple(z["rshape"]))
        _REF["path"] = path
    b = _REF["R"][:, col].toarray().ravel()
    t0 = time.perf_counter()
    x, info = cg(_REF["A"], b, rtol=tol, maxiter=maxiter)
    return time.perf_counter() - t0, info


def run_reference(args):
    """The reference's CPU path for this workload on the host cores (the
    oracle port; the reference itself is Python and is not present on the
    GPU machine): femsolve(method='cg') per column in a process pool, like
    redbirdpy's _iterative_parallel (solver.py:310-377), one column per core
    per step, reference defaults tol 1e-10 / maxiter 1000."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import multiprocessing as mp
    import tempfile

    from oracle import femoracle as fo

    cfg = workload_cfg()
    ocfg, _ = fo.meshprep(cfg)
    A = fo.femlhs(ocfg, fo.deldotdel(ocfg["node"], ocfg["elem"], ocfg["evol"]))
    rhs, _, _, _ = fo.femrhs(ocfg)
    ncore = os.cpu_count() or 1
    tmp = os.path.join(tempfile.gettempdir(), f"rb_ref_{os.getpid()}.npz")
    rc = rhs.tocsc()
    np.savez(tmp, data=A.data, indices=A.indices, indptr=A.indptr, rdata=rc.data, rindices=rc.indices,
             rindptr=rc.indptr, rshape=np.array(rc.shape))
    ctx = mp.get_context("spawn")
    times = []
    # one BLAS thread per worker process (the pool provides the parallelism)
    for var in ("OMP_NUM_THREADS", "OPENBLAS_NUM_THREADS", "MKL_NUM_THREADS"):
        os.environ[var] = "1"
    with ctx.Pool(ncore, initializer=_ref_init) as pool:
        pool.map(_ref_worker, [(tmp, j % 128, 1e-10, 1) for j in range(ncore)])  # load the system per worker
        col = 0
        for s in range(args.warmup + args.steps):
            jobs = [(tmp, (col + j) % 128, 1e-10, 1000) for j in range(ncore)]
            col += ncore
            t0 = time.perf_counter()
            res = pool.map(_ref_worker, jobs)
            dt = time.perf_counter() - t0
            if s >= args.warmup:
                times.append(dt)
                infos = [r[1] for r in res]
    os.remove(tmp)
    ms = 1e3 * float(np.mean(times))
    v = ncore / (ms * 1e-3)
    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": round(v, 5), "unit": UNIT, "n_gpus": 0,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 1), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": "box 100x100x50 mm, 1 mm Kuhn (520251 nodes, 3000000 tets), 64 src + 64 det, CW",
                   "solver": "scipy CG per column (reference femsolve method='cg'), tol 1e-10, maxiter 1000",
                   "columns_converged": f"{sum(1 for i in infos if i == 0)} of {len(infos)} in the last step "
                                        "(the rest stop at maxiter, as the reference does)"},
        "cpu_baseline": {"value": round(v, 5), "unit": UNIT, "cores": ncore, "kind": "port",
                         "sample": f"{ncore} columns per step, one per core"},
        "e2e": {"value": round(v, 5), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--no-gn", action="store_true", help="skip the Gauss-Newton iteration measurement")
    ap.add_argument("--no-fp64-gn", action="store_true", help="skip the plain-FP64 GN comparison")
    ap.add_argument("--no-adjoint", action="store_true", help="skip the adjoint-gradient / Jacobian measurement")
    ap.add_argument("--no-batch", action="store_true", help="skip the batched-instances measurement")
    ap.add_argument("--profile-run", action="store_true", help="short fixed workload for ncu captures")
    ap.add_argument("--spacing", type=float, default=1.0, help="mesh pitch (mm) of --profile-run")
    ap.add_argument("--with-gn", action="store_true", help="--profile-run: add one GN iteration")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    elif args.profile_run:
        run_profile(args)
    else:
        run_b200(args)


if __name__ == "__main__":
    main()
