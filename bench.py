#!/usr/bin/env python
"""Benchmark: batched eigensolves on B200 (the headline) with the plain GPU Lanczos beside it.

Workload (synthetic, seeded; no dataset): 3x9 k-mesh, Ne=9 -> 27 momentum sectors of ~174k
states.  H(U0) = H0 + U0 V (one-body band + random-phase two-body recipe, seed 2) with 32
interaction strengths U0 evenly spaced in [0.5, 2.0]; the 4 lowest eigenpairs of each
(sector, U0) to <= 1e-10 relative eigenvalue error.

A step is one sector x 32 U0 values = 32 solves through the batched mixed-precision solver
(c64 block matvec, FP64 recurrences, FP64 Rayleigh-Ritz).  `value` times K steps with the
sector bases already in HBM (enumerated by the basis kernel before timing); `e2e` times the
same steps through the public API with host buffers (basis + operator in, eigenvalues and
eigenvectors out).  The plain comparison solves U0 values of one sector one at a time with the
FP64 single-vector Lanczos.

Serving (rank 0, N = 1): a Poisson stream of solve requests at 50 req/s (seed 4; mesh uniform
over --serve-meshes, uniform sector, U0 ~ U(0.5, 2), nev 1..20, tol 1e-10) through the
continuous-batching server, and the same requests solved one at a time by the plain FP64 GPU
Lanczos, both live against the arrival clock; latency is arrival -> eigenvalues on the host.
Queued requests on the same sector are solved together by the server (continuous batching).
The 4x9 Ne=12 mesh (~35M states per sector) is left out of the default stream because one of
its solves alone takes tens of seconds; --serve-meshes 3x5,3x9,3x10,4x9 includes it.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
Under torchrun (N > 1) every rank runs its own sectors (replicas, no data-path collective).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "momentumed.jl_b200"))

MESH = (3, 9)
NE = 9
SEED = 2
NEV = 4
NU = 32
KRYLOV = 30
# DRAM bytes (read + write) of one c64 x32 block-map launch on this workload, from an ncu capture
# of `bench.py --profile-only` (dram__bytes_read.sum + dram__bytes_write.sum = 46.5 + 28.8 MB): the
# x block and the term tables stay in L2, so the per-hit gathers of the algorithmic count hit L2.
MV_DRAM_BYTES = 75.3e6
# DRAM bytes (read + write) of one launch of the c64 x32 block map over the hit cache on this
# workload, from an ncu capture of `bench.py --profile-only` (381.3 + 32.5 MB): the hit stream,
# x and y once and the row metadata; the x-row gathers (9.6 GB per launch) are served by L2.
MV_DRAM_BYTES_HC = 413.8e6
METRIC = "batched solves/s, p50/p99 latency vs plain GPU Lanczos at <=1e-10 eig error"


def workload_name() -> str:
    return (f"3x9 mesh Ne=9, one sector (~174k states) x {NU} U0 in [0.5,2] per step, nev={NEV}, "
            f"krylovdim={KRYLOV}, tol 1e-12")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--plain", type=int, default=4, help="U0 values solved one at a time for the plain comparison")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline")
    ap.add_argument("--krylovdim", type=int, default=0, help="Krylov dimension of the batched solver (default 30)")
    ap.add_argument("--profile-only", action="store_true", help="one short run for ncu (no timing output)")
    ap.add_argument("--workload", default="batch_3x9",
                    choices=["batch_3x9", "plain_3x5", "plain_3x9", "plain_3x10", "two_comp_4x6"],
                    help="batch_3x9 (the headline); the others time plain single-vector solves")
    ap.add_argument("--no-serve", action="store_true", help="skip the serving stream")
    ap.add_argument("--sparse-batch", type=int, default=1,
                    help="also time the headline sweep on the sparse method (1) or not (0)")
    ap.add_argument("--method", default="map", choices=["map", "sparse"],
                    help="plain workloads (and --profile-only of the sweep): matrix-free map, or the sparse "
                         "method (device-built CSR + SpMV)")
    ap.add_argument("--serve-requests", type=int, default=80)
    ap.add_argument("--serve-meshes", default="3x5,3x9,3x10", help="subset of 3x5,3x9,3x10,4x9")
    ap.add_argument("--serve-slots", type=int, default=4)
    ap.add_argument("--serve-hbm-gb", type=float, default=100.0)
    ap.add_argument("--serve-policy", default="", help="served arm switches: alone=fp64|mixed,sparse=1|0,hitcache=1|0,large=<concurrent large solves>,"
                         "group=<smallest group>")
    ap.add_argument("--serve-only", action="store_true", help="only the serving stream (one JSON object)")
    return ap.parse_args()


def workload_operators():
    """(para, pair arrays (amp_a, amp_b, in, out, pm), u grid) of the sweep."""
    import momed
    from momed.core import pair_operator
    from momed.synthetic import mesh_para, u_grid

    para, _ = mesh_para(*MESH, SEED)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    return para, pair_operator(A, B), u_grid(NU, 0.5, 2.0)


# ----------------------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *a):
        self.lines = []
        if self.proc:
            self.proc.terminate()
            try:
                out, _ = self.proc.communicate(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
                out, _ = self.proc.communicate()
            self.lines = [l for l in out.splitlines() if l.strip()]

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in getattr(self, "lines", []):
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


# ----------------------------------------------------------------------------- distributed
_DIST_DEVICE = "cuda"


def dist_setup(args, backend: str = "nccl"):
    """One process per GPU (RANK / LOCAL_RANK / WORLD_SIZE / MASTER_* from the launcher).  The
    ranks only exchange timings and counts (replicas: no data-path collective); `backend`
    "gloo" runs the same plumbing on CPU."""
    global _DIST_DEVICE
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        if backend == "nccl":
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600),
                                    device_id=torch.device("cuda", local))
            _DIST_DEVICE = "cuda"
        else:
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=120))
            _DIST_DEVICE = "cpu"
    return rank, world, local


def sector_order(rank: int, world: int, nsec: int, count: int):
    """The sectors rank `rank` solves, in order: every world-th sector starting at rank, cycling."""
    return [(rank + world * i) % nsec for i in range(count)]


def all_max(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=_DIST_DEVICE)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def all_sum(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=_DIST_DEVICE)
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def barrier(world: int):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


# ----------------------------------------------------------------------------- CPU arm
def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    return O


# maps in one bounded sample of the reference arm (the first Krylov cycle of a solve, cut short)
REF_SAMPLE_MAPS = 12


def cpu_reference_solve(basis, pair, u0, nthreads, maxiter=100, krylovdim=None):
    """The reference's CPU path restated (oracle): gather map over the full term list + FP64 Lanczos."""
    O = _oracle()
    amp_a, amp_b, in_, out, pm = pair
    full = np.zeros(len(amp_a), O.SCAT_DTYPE)
    amp = amp_a + u0 * amp_b
    full["re"], full["im"], full["out"], full["in"], full["pm"] = amp.real, amp.imag, out, in_, pm
    t0 = time.perf_counter()
    vals, _, _, info = O.eigsolve(basis, full, NEV, krylovdim=krylovdim or KRYLOV, tol=1e-12, maxiter=maxiter,
                                  seed=1, nthreads=nthreads, want_vectors=True)
    return time.perf_counter() - t0, vals, info


def reference_workload():
    """Sector bases and the operator pair of the sweep, built by the oracle alone (the reference's
    host algorithms restated in C): no code of this package runs in the reference arm."""
    O = _oracle()
    a, b = MESH
    bases, _ = O.momentum_subspaces(O.mesh_klist(a, b), (a, b), (NE,))
    S = O.Synth(a, b, SEED)
    one = O.hermitian_complete(O.sort_merge(S.onebody()))
    two = O.hermitian_complete(O.sort_merge(S.twobody()))
    # H(u) = H0 + u V on the union of the two completed term lists (one-body terms are diagonal)
    keys = np.concatenate([one[["out", "in"]], two[["out", "in"]]])
    uk, inv = np.unique(keys, return_inverse=True)
    amp_a = np.zeros(len(uk), np.complex128)
    amp_b = np.zeros(len(uk), np.complex128)
    np.add.at(amp_a, inv[:len(one)], one["re"] + 1j * one["im"])
    np.add.at(amp_b, inv[len(one):], two["re"] + 1j * two["im"])
    pm = np.zeros(len(uk), np.uint64)
    pm[inv[:len(one)]] = one["pm"]
    pm[inv[len(one):]] = two["pm"]
    u = 0.5 + 1.5 * np.arange(NU) / (NU - 1)
    return bases, (amp_a, amp_b, uk["in"].copy(), uk["out"].copy(), pm), u


def run_reference(args, rank, world):
    """--impl reference: the reference's CPU path (the oracle's C restatement of the CPU map
    linear_map.jl:100-118 and the FP64 Lanczos, all host threads) on this workload.  Rank 0 alone
    runs.  A full solve takes a minute or more on the host, so each step is a bounded sample: the
    first REF_SAMPLE_MAPS Lanczos steps (maps with full reorthogonalisation) of the FP64 solve of
    the step's (sector, U0) pair, the sectors and U0 values in the order of the GPU arm's steps.
    solves/s = the sampled map rate / the maps of one full solve, counted by one complete solve of
    the first timed pair before the steps (its own rate is reported beside)."""
    if rank != 0:
        return
    bases, pair, u = reference_workload()
    nsec = len(bases)
    nthreads = os.cpu_count() or 1
    W, K = max(args.warmup, 0), max(args.steps, 1)
    order = sector_order(0, 1, nsec, W + K)
    full_t, full_vals, full_info = cpu_reference_solve(bases[order[W]], pair, float(u[W % NU]), nthreads)
    mv_full = full_info["matvecs"]
    for i in range(W):
        cpu_reference_solve(bases[order[i]], pair, float(u[i % NU]), nthreads, maxiter=0, krylovdim=REF_SAMPLE_MAPS)
    times, mvs = [], []
    for i in range(K):
        dt, _, info = cpu_reference_solve(bases[order[W + i]], pair, float(u[(W + i) % NU]), nthreads, maxiter=0,
                                          krylovdim=REF_SAMPLE_MAPS)
        times.append(dt)
        mvs.append(info["matvecs"])
    mv_rate = sum(mvs) / sum(times)
    value = mv_rate / mv_full
    line = {
        "impl": "reference", "metric": METRIC, "value": value,
        "unit": "solves/s", "n_gpus": 0, "steps": K, "warmup": W,
        "ms_per_step": 1e3 * sum(times) / K, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "c128", "data": "synthetic",
        "config": {"workload": workload_name(),
                   "solver": "reference CPU map + FP64 Lanczos (oracle restatement), one (sector, U0) pair per "
                             "step in the GPU arm's order",
                   "step_sample": f"first {REF_SAMPLE_MAPS} Lanczos steps of the pair's FP64 solve (maps with "
                                  f"full reorthogonalisation); solves/s = map rate / {mv_full} maps per full solve",
                   "full_solve": {"seconds": full_t, "matvecs": mv_full, "solves_per_s": 1.0 / full_t,
                                  "converged": full_info["converged"]}},
        "cpu_baseline": {"value": value, "unit": "solves/s", "cores": nthreads, "kind": "port",
                         "sample": f"{K} samples of {REF_SAMPLE_MAPS} Lanczos steps ({sum(mvs)} maps) of (sector, U0) solves of "
                                   f"{len(bases[order[W]])}-state sectors, scaled by one full solve's "
                                   f"{mv_full} maps"},
        "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ----------------------------------------------------------------------------- serving
def serve_krylovdim(nev: int) -> int:
    return max(KRYLOV, 2 * nev + 12)


def serve_bench(args, device: int):
    """Serving form: the Poisson request stream through momed_serve_* (mixed precision,
    `args.serve_slots` slots; queued requests on one sector are solved together) and the same
    requests solved one at a time by the plain FP64 GPU Lanczos, both live against the arrival
    clock.  At 50 req/s the queue outgrows either server within the first second, so solves/s
    is the service capacity.  Latency is arrival -> eigenvalues on the host."""
    import momed
    from momed import _lib
    from momed.core import pair_operator
    from momed.synthetic import SERVE_MESHES, mesh_para, serve_requests

    meshes = [m for m in args.serve_meshes.split(",") if m]
    h = momed.Handle(device)
    sectors, ops = {}, {}
    for m in meshes:
        ne, seed = SERVE_MESHES[m]
        a, b = (int(x) for x in m.split("x"))
        para, _ = mesh_para(a, b, seed)
        sectors[m] = [s[1] for s in h.enumerate_basis(para.k_list, para.Gk, 1, 1, (ne,))]
        A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
        B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
        ops[m] = pair_operator(A, B)
    reqs = serve_requests(args.serve_requests, meshes, {m: len(sectors[m]) for m in meshes})

    def pct(x, q):
        return float(np.percentile(np.asarray(x), q)) if len(x) else None

    # plain: one request at a time, FP64 single-vector Lanczos, live against arrivals; once with
    # the matrix-free map and once with the sparse method (the matrix built for each request)
    def run_plain(sparse, block=False):
        # the plain GPU Lanczos is the reference's algorithm on the device: single-vector Krylov
        # over the map that evaluates every term at every application (no hit cache);
        # block=True runs the library's default solver one at a time (over the hit cache)
        if block:
            os.environ.pop("MOMED_BLOCK", None)
            os.environ.pop("MOMED_HITCACHE", None)
        else:
            os.environ["MOMED_BLOCK"] = "0"
            os.environ["MOMED_HITCACHE"] = "0"
        vals_, lat_, service_ = [], [], []
        cur = None
        t0 = time.perf_counter()
        for r in reqs:
            now = time.perf_counter() - t0
            if now < r["arrival"]:
                time.sleep(r["arrival"] - now)
            s0 = time.perf_counter()
            if cur != r["mesh"]:
                h.set_scatter_pair(*ops[r["mesh"]])
                cur = r["mesh"]
            h.set_basis(sectors[r["mesh"]][r["sector"]])
            h.set_param(r["u"])
            if sparse:
                h.build_sparse()
            v, _, _, _ = h.eigsolve(r["nev"], krylovdim=serve_krylovdim(r["nev"]), tol=r["tol"], maxiter=300,
                                    want_vectors=False, precision=_lib.PREC_FP64)
            s1 = time.perf_counter()
            vals_.append(v)
            service_.append(s1 - s0)
            lat_.append(s1 - t0 - r["arrival"])
        span = time.perf_counter() - t0
        os.environ.pop("MOMED_BLOCK", None)
        os.environ.pop("MOMED_HITCACHE", None)
        return vals_, lat_, service_, span

    plain_vals, plain_lat, plain_service, plain_span = run_plain(False)
    sp_vals, sp_lat, sp_service, sp_span = run_plain(True)
    bl_vals, bl_lat, bl_service, bl_span = run_plain(False, block=True)
    h.close()
    # serving policy switches (MOMED_SERVE_ALONE=fp64|mixed, MOMED_SERVE_SPARSE=1|0,
    # MOMED_SERVE_HITCACHE=1|0) for the served arm
    for kv in [x for x in args.serve_policy.split(",") if x]:
        k, v = kv.split("=")
        os.environ[{"alone": "MOMED_SERVE_ALONE", "sparse": "MOMED_SERVE_SPARSE", "hitcache": "MOMED_SERVE_HITCACHE",
                    "large": "MOMED_SERVE_LARGE_MAX", "group": "MOMED_SERVE_MIN_GROUP"}[k]] = v

    def run_server():
        srv = momed.Server(device, slots=args.serve_slots, hbm_budget=int(args.serve_hbm_gb * (1 << 30)))
        op_id = {m: srv.register_operator(*ops[m]) for m in meshes}
        ids = []
        t0 = time.perf_counter()
        for r in reqs:
            now = time.perf_counter() - t0
            if now < r["arrival"]:
                time.sleep(r["arrival"] - now)
            ids.append(srv.submit(op_id[r["mesh"]], sectors[r["mesh"]][r["sector"]], r["u"], r["nev"], tol=r["tol"],
                                  krylovdim=serve_krylovdim(r["nev"]), maxiter=300, precision=_lib.PREC_MIXED))
        vals, lat, conv, groups = [], [], [], {}
        for rid, r in zip(ids, reqs):
            while True:
                st, v, res, info, q, l = srv.poll(rid, r["nev"], wait_ms=1000)
                if st >= 2:
                    break
            vals.append(v)
            lat.append(l)
            conv.append(info["converged"] >= r["nev"])
            g = groups.setdefault((r["mesh"], r["sector"], info["matvecs"], info["seconds"]), [])
            g.append(r["nev"])
        span = time.perf_counter() - t0
        srv.stop()
        return vals, lat, conv, span, groups

    s_vals, s_lat, s_conv, s_span, groups = run_server()
    n_solves = len(groups)
    slow = sorted(groups.items(), key=lambda kv: -kv[0][3])[:6]
    gsizes = {}
    for k, v in groups.items():
        gsizes[len(v)] = gsizes.get(len(v), 0) + 1
    errs = [float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0))) for a, b in zip(s_vals, plain_vals)]
    n = len(reqs)
    sizes = {m: [len(x) for x in sectors[m]] for m in meshes}
    return {
        "stream": f"{n} requests, Poisson 50 req/s (seed 4), meshes {meshes}, uniform sector, U0~U(0.5,2), "
                  f"nev 1..20, tol 1e-10",
        "meshes_states_per_sector": {m: [min(v), max(v)] for m, v in sizes.items()},
        "served": {"solves_per_s": n / s_span, "latency_ms_p50": 1e3 * pct(s_lat, 50),
                   "latency_ms_p99": 1e3 * pct(s_lat, 99), "slots": args.serve_slots,
                   "device_solves": n_solves, "group_sizes": {str(k): v for k, v in sorted(gsizes.items())},
                   "slowest_solves": [{"mesh": k[0], "nev": v, "device_s": round(k[3], 3), "matvecs": k[2]}
                                      for k, v in slow],
                   "precision": "mixed requests: the batched mixed solver, for groups on one sector and "
                                "(one right-hand side) for a request alone; maps over the hit cache when "
                                "it fits the budget, else the sparse method when its matrix fits",
                   "all_converged": bool(all(s_conv)), "max_rel_eig_err_vs_plain_fp64": max(errs)},
        "plain_one_at_a_time": {"solves_per_s": n / plain_span, "latency_ms_p50": 1e3 * pct(plain_lat, 50),
                                "latency_ms_p99": 1e3 * pct(plain_lat, 99),
                                "service_ms_p50": 1e3 * pct(plain_service, 50), "precision": "fp64",
                                "method": "map evaluating every term at every application (no hit cache), "
                                          "single-vector Lanczos"},
        "plain_sparse_one_at_a_time": {"solves_per_s": n / sp_span, "latency_ms_p50": 1e3 * pct(sp_lat, 50),
                                       "latency_ms_p99": 1e3 * pct(sp_lat, 99),
                                       "service_ms_p50": 1e3 * pct(sp_service, 50), "precision": "fp64",
                                       "method": "sparse (matrix built per request), single-vector Lanczos",
                                       "max_rel_eig_err_vs_map": max(
                                           float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0)))
                                           for a, b in zip(sp_vals, plain_vals))},
        "solver_one_at_a_time": {"solves_per_s": n / bl_span, "latency_ms_p50": 1e3 * pct(bl_lat, 50),
                                 "latency_ms_p99": 1e3 * pct(bl_lat, 99),
                                 "service_ms_p50": 1e3 * pct(bl_service, 50), "precision": "fp64",
                                 "method": "the library's default solver on the map: single-vector Lanczos "
                                           "over the hit cache (block Lanczos where no cache fits)",
                                 "max_rel_eig_err_vs_map": max(
                                     float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0)))
                                     for a, b in zip(bl_vals, plain_vals))},
        "policy": args.serve_policy or "default (alone: the request's precision; hit cache, else sparse method, when it fits)",
        "speedup_served_vs_plain": (n / s_span) / (n / plain_span),
        "speedup_served_vs_plain_sparse": (n / s_span) / (n / sp_span),
    }


# ----------------------------------------------------------------------------- plain workloads
def mv_bytes(N: int, nnz: int, nscat: int, s: int) -> float:
    """Algorithmic bytes of one single-vector map: basis keys, x stream read and y write, one
    gather per (row, term) hit, and the term list (amplitude and three masks per term)."""
    return N * (8 + 2 * s) + nnz * s + nscat * (s + 24)


def block_size(nev: int, N: int) -> int:
    """Block size the FP64 eigensolver picks for nev pairs on N states (0: single-vector Lanczos;
    block_size_for in block_lanczos.cu)."""
    if os.environ.get("MOMED_BLOCK"):
        b = int(os.environ["MOMED_BLOCK"])
        return b if b in (4, 8, 16) and N >= 16 * b else 0
    cached = os.environ.get("MOMED_HITCACHE", "") != "0"   # the bench sectors' hit caches all fit
    if nev < 6 or N < (2000000 if cached else 500000):
        return 0
    return 4 if nev <= 10 else 8


def sp_bytes(N: int, nnz_sp: int, s: int) -> float:
    """Algorithmic HBM bytes of one CSR SpMV: the column and value of every stored entry, the row
    pointers, and x and y once each (x, at most a few tens of MB here, serves its gathers from L2)."""
    return nnz_sp * (4 + s) + N * (8 + 2 * s)


def run_plain_workload(args, rank, world, local):
    """--workload plain_3x5 | plain_3x9 | plain_3x10 | two_comp_4x6: one sector per step solved by the plain
    single-vector Lanczos (FP64, c128 map; the mixed-precision solve is timed beside it).
    --method sparse: the sparse method instead, each step building the sector's CSR matrix on
    the device and solving with the CSR SpMV (build inside the timed step, as in EDsolve)."""
    import torch

    import momed
    from momed import _lib
    from momed.core import pair_operator
    from momed.synthetic import WORKLOADS, mesh_para

    w = WORKLOADS[args.workload]
    ncc = w["Nc_conserve"]
    para, _ = mesh_para(w["a"], w["b"], w["seed"], Nc_conserve=ncc)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    pair = pair_operator(A, B)
    nev, kd = w["nev"], w.get("krylovdim", 30)
    torch.cuda.set_device(local)
    h = momed.Handle(local)
    stream = torch.cuda.Stream(device=local)
    h.set_stream(stream.cuda_stream)
    sectors = h.enumerate_basis(para.k_list, para.Gk, 1, ncc, w["N_each"])
    h.set_scatter_pair(*pair)
    h.set_param(1.0)
    W, K = max(args.warmup, 0), max(args.steps, 1)
    order = sector_order(rank, world, len(sectors), W + K)

    sparse = args.method == "sparse"

    def solve(sidx, prec):
        h.select_sector(sidx, len(sectors[sidx][1]))
        if sparse:
            h.build_sparse()
        return h.eigsolve(nev, krylovdim=kd, tol=1e-12, seed=1, want_vectors=False, precision=prec)

    if args.profile_only:
        solve(order[0], _lib.PREC_FP64)
        return
    for i in range(W):
        solve(order[i], _lib.PREC_FP64)
    torch.cuda.synchronize()
    launches0 = _lib.kernel_launches()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(K + 1)]
    infos, vals64 = [], []
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        ev[0].record(stream)
        for i in range(K):
            v, _, _, info = solve(order[W + i], _lib.PREC_FP64)
            ev[i + 1].record(stream)
            infos.append(info)
            vals64.append(v)
        torch.cuda.synchronize()
    barrier(world)
    step_ms = [ev[i].elapsed_time(ev[i + 1]) for i in range(K)]
    launches = _lib.kernel_launches() - launches0
    # device time of the maps: the first (up to 3) timed sectors again with per-launch events, which
    # need separate launches (the timed solves run their steps as cooperative kernels, some with the
    # map inside)
    h.profile(True)
    for i in range(min(K, 3)):
        solve(order[W + i], _lib.PREC_FP64)
    torch.cuda.synchronize()
    n_mv, ms_mv = h.profile_read(_lib.KERNEL_SPMV_C128 if sparse else _lib.KERNEL_MATVEC_C128)
    n_bmv, ms_bmv = h.profile_read(_lib.KERNEL_BLOCK_MATVEC_C128)
    n_hmv, ms_hmv = h.profile_read(_lib.KERNEL_HC_MATVEC_C128)
    n_hbmv, ms_hbmv = h.profile_read(_lib.KERNEL_HC_BLOCK_C128)
    h.profile(False)
    use_hc = not sparse and (n_hmv + n_hbmv) > 0      # the solves ran over the map's hit cache
    if use_hc:
        n_mv, ms_mv, n_bmv, ms_bmv = n_hmv, ms_hmv, n_hbmv, ms_hbmv
    # nev >= 2 on large sectors runs the block solver (block_size_for in block_lanczos.cu): its maps
    # are block maps of B right-hand sides, the single-vector launches only the final residual maps
    bsz = block_size(nev, len(sectors[order[W]][1])) if not sparse else 0
    if bsz and n_bmv > 0:
        n_mv, ms_mv = n_bmv, ms_bmv
    else:
        bsz = 0                                        # over the pair tables: the single-vector solver
    elapsed = all_max(sum(step_ms) / 1e3, world)
    value = all_sum(K, world) / elapsed
    nb, nnz_mean, build_ms, hc_info = [], [], [], []
    for i in range(K):
        sidx = order[W + i]
        h.select_sector(sidx, len(sectors[sidx][1]))
        st = h.stats()
        if use_hc:
            hc = h.build_hit_cache()
            hc_info.append(hc)
            pairs = 0 if bsz else pair_table_bytes(hc, sum(w["N_each"]), len(sectors[sidx][1]))
            nb.append(pair_bytes(pairs, sum(w["N_each"]), len(sectors[sidx][1]), 16) if pairs > 0 else
                      hc_bytes(len(sectors[sidx][1]), hc["hits"], len(pair[0]), max(bsz, 1), 16))
            nnz_mean.append(st["nnz"])
        elif sparse:
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            nsp = h.build_sparse()
            build_ms.append((time.perf_counter() - t0) * 1e3)
            nb.append(sp_bytes(len(sectors[sidx][1]), nsp, 16))
            nnz_mean.append(nsp)
        elif bsz:
            nb.append(block_bytes(len(sectors[sidx][1]), st["nnz"], len(pair[0]), bsz, 16))
            nnz_mean.append(st["nnz"])
        else:
            nb.append(mv_bytes(len(sectors[sidx][1]), st["nnz"], len(pair[0]), 16))
            nnz_mean.append(st["nnz"])
    # the mixed-precision solve of the same sectors, for comparison
    t_mixed, err_mixed = [], []
    for i in range(K):
        t0 = time.perf_counter()
        v, _, _, _ = solve(order[W + i], _lib.PREC_MIXED)
        t_mixed.append(time.perf_counter() - t0)
        err_mixed.append(float(np.max(np.abs(v - vals64[i]) / np.maximum(np.abs(vals64[i]), 1.0))))
    # e2e: the same solves through the public API with host buffers (basis in, values + vectors out)
    e2e_t, h2d, d2h = [], [], []
    for i in range(K):
        basis = sectors[order[W + i]][1]
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        h.set_basis(basis)
        if sparse:
            h.build_sparse()
        v, vecs, _, _ = h.eigsolve(nev, krylovdim=kd, tol=1e-12, seed=1, want_vectors=True,
                                   precision=_lib.PREC_FP64)
        e2e_t.append(time.perf_counter() - t0)
        h2d.append(basis.nbytes)
        d2h.append(v.nbytes + vecs.nbytes)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu and not sparse:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O
        amp = pair[0] + pair[1]
        full = np.zeros(len(amp), O.SCAT_DTYPE)
        full["re"], full["im"], full["out"], full["in"], full["pm"] = amp.real, amp.imag, pair[3], pair[2], pair[4]
        basis = sectors[order[W]][1]
        x = np.random.default_rng(0).standard_normal(len(basis)) + 0j
        nthreads = os.cpu_count() or 1
        t0, reps = time.perf_counter(), 0
        while time.perf_counter() - t0 < 10.0 or reps == 0:
            O.matvec(basis, full, x, nthreads=nthreads)
            reps += 1
        cpu_mv = (time.perf_counter() - t0) / reps
        mv_per_solve = float(np.mean([i["matvecs"] for i in infos]))
        cpu = {"value": 1.0 / (cpu_mv * mv_per_solve), "unit": "solves/s", "cores": nthreads, "kind": "port",
               "sample": f"{reps} CPU maps of one {len(basis)}-state sector (reference CPU map restated, "
                         f"{cpu_mv * 1e3:.0f} ms each) x {mv_per_solve:.0f} maps per solve (the GPU solve's count)"}
    if rank == 0:
        avg_ms = ms_mv / max(n_mv, 1)
        achieved = float(np.mean(nb)) / (avg_ms * 1e-3) / 1e9
        peaks_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
        peak, peak_src = 6650.0, "fallback"
        if os.path.exists(peaks_path):
            try:
                peak = float(json.load(open(peaks_path))["hbm_gbs"])
                peak_src = "measured"
            except Exception:
                pass
        N0 = len(sectors[order[W]][1])
        metric = ("solves/s (sparse method: device-built CSR matrix + FP64 single-vector Lanczos, one sector "
                  "per step)" if sparse else
                  f"solves/s (plain FP64 {'block' if bsz else 'single-vector'} Lanczos, one sector per step)")
        if sparse:
            kernel = "CSR SpMV c128 (k_spmv<double>)"
            extra = {"sparse": {"build_ms_mean": float(np.mean(build_ms)), "entries_mean": float(np.mean(nnz_mean)),
                                "matrix_bytes_per_entry": 28,
                                "algorithmic_bytes": "column + c128 value per entry, row pointers, x and y once "
                                                     "(x gathers served from L2)"}}
        elif bsz:
            kernel = (f"block map c128 x{bsz} over the hit cache (k_block_hc<double, {bsz}>, block Lanczos)" if use_hc
                      else f"block map c128 x{bsz} (k_block_matvec_v<double, {bsz}>, block Lanczos)")
            extra = {"block_lanczos": {"block": bsz, "maps_per_launch": bsz}}
        else:
            kernel = ("map c128 over the pair tables (k_pair_ids, k_pair_rows)" if use_hc and pairs > 0 else
                      "map c128 over the hit cache (k_matvec_hc<double>)" if use_hc else "map c128 (k_matvec<double>)")
            extra = {}
        if use_hc:
            extra["hit_cache"] = {"hits_per_sector": float(np.mean([c["hits"] for c in hc_info])),
                                  "bytes_per_sector": float(np.mean([c["bytes"] for c in hc_info])),
                                  "build_ms": float(np.mean([c["build_ms"] for c in hc_info])),
                                  "note": "built inside each timed solve (first map of the sector)"}
        line = {
            "metric": metric, "value": value,
            "unit": "solves/s", "n_gpus": world, "steps": K, "warmup": W, "ms_per_step": elapsed * 1e3 / K,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic",
            "config": {"workload": f"{args.workload}: {w['a']}x{w['b']} mesh, N_each={w['N_each']}, "
                                   f"~{N0} states per sector, nev={nev}, krylovdim={kd}, tol 1e-12",
                       "parallelism": f"replicas x{world}", "l2": "a step streams the Krylov basis (> L2)"},
            "latency_ms": {"p50": float(np.percentile(step_ms, 50)), "p99": float(np.percentile(step_ms, 99))},
            "matvecs_per_s": float(np.mean([i["matvecs"] for i in infos])) * value,
            "mixed_precision": {"solves_per_s": K / sum(t_mixed), "max_rel_eig_err_vs_fp64": max(err_mixed)},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": None, "peak_source": peak_src,
                         "kernel": kernel, "launches": n_mv, "avg_launch_ms": avg_ms,
                         "algorithmic_bytes_per_launch": float(np.mean(nb)), "nnz": float(np.mean(nnz_mean))},
            "cpu_baseline": cpu,
            "e2e": {"value": K / sum(e2e_t), "unit": "solves/s", "h2d_bytes_per_step": int(np.mean(h2d)),
                    "d2h_bytes_per_step": int(np.mean(d2h))},
            "gpu_launches": int(all_sum(launches, world)),
            "clocks": clk.summary(),
        }
        line.update(extra)
        print(json.dumps(line), flush=True)
    h.close()


# ----------------------------------------------------------------------------- our arm
def hc_bytes(N: int, hits: int, nscat: int, nb: int, s: int) -> float:
    """Algorithmic bytes of one map launch over the hit cache: each row's hit range, run ends and
    diagonal sums (A and B parts), x read and y written for nb right-hand sides, one 8-byte hit
    record and one nb-wide gather per off-diagonal hit, and the amplitude table (A and B) once."""
    return N * (16 + 2 * s + 2 * s * nb) + hits * (8 + s * nb) + nscat * 2 * s


def pair_table_bytes(info: dict, ne: int, N: int) -> int:
    """Size of the pair tables of a freshly built cache, which has them with a workspace of 16 bytes for
    every pair of every row, or the hit records (8 bytes per hit, 64 per row); 0 for those."""
    records = info["hits"] * 8 + (N + 1) * 8 + N * 56
    return info["bytes"] - N * (ne * (ne - 1) // 2) * 16 if info["mode"] == "full" and info["bytes"] != records else 0


def pair_bytes(tables: int, ne: int, N: int, s: int) -> float:
    """Algorithmic bytes of one map application over the pair tables: the tables once, psi written and
    read and x gathered for every pair of every row, x and y once for the diagonal."""
    return tables + N * (ne * (ne - 1) // 2) * 3 * s + N * (8 + 2 * s)


def block_bytes(N: int, nnz: int, nscat: int, nb: int, s: int) -> float:
    """Algorithmic bytes of one block matvec launch: basis keys, x stream read and y write for nb
    right-hand sides, one nb-wide gather per (row, term) hit, and the term list (two amplitudes
    and three masks per term)."""
    return N * (8 + 2 * s * nb) + nnz * s * nb + nscat * (2 * s + 24)


def main():
    global KRYLOV
    args = parse()
    if args.krylovdim > 0:
        KRYLOV = args.krylovdim
    rank, world, local = dist_setup(args)
    if args.impl == "reference":
        run_reference(args, rank, world)
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
        return
    if args.serve_only:
        if rank == 0:
            import torch
            torch.cuda.set_device(local)
            print(json.dumps({"serving": serve_bench(args, local)}), flush=True)
        return
    if args.workload != "batch_3x9":
        run_plain_workload(args, rank, world, local)
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
        return
    import torch

    import momed
    from momed import _lib

    torch.cuda.set_device(local)
    para, pair, u = workload_operators()
    amp_a, amp_b, in_, out, pm = pair
    h = momed.Handle(local)
    stream = torch.cuda.Stream(device=local)
    h.set_stream(stream.cuda_stream)
    sectors = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (NE,))        # kernel (a), outside timing
    nsec = len(sectors)
    h.set_scatter_pair(amp_a, amp_b, in_, out, pm)
    W, K = max(args.warmup, 0), max(args.steps, 1)
    order = sector_order(rank, world, nsec, W + K)

    def step_device(sidx):
        h.select_sector(sidx, len(sectors[sidx][1]))
        vals, _, res, info = h.batch_solve(u, NEV, krylovdim=KRYLOV, tol=1e-12, precision=_lib.PREC_MIXED)
        return vals, res, info

    if args.profile_only:
        if args.method == "sparse":            # one step of the sweep on the sparse method
            h.select_sector(order[0], len(sectors[order[0]][1]))
            h.build_sparse()
            h.batch_solve(u, NEV, krylovdim=KRYLOV, tol=1e-12, precision=_lib.PREC_MIXED)
            h.release_sparse()
        else:
            step_device(order[0])
        return

    for i in range(W):
        step_device(order[i])
    torch.cuda.synchronize()
    # ---------------------------------------------------------------- value: inputs resident in HBM
    launches0 = _lib.kernel_launches()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(K + 1)]
    per_step_nnz, per_step_n, infos, all_vals = [], [], [], []
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        ev[0].record(stream)
        for i in range(K):
            sidx = order[W + i]
            vals, res, info = step_device(sidx)
            ev[i + 1].record(stream)
            infos.append(info)
            all_vals.append((sidx, vals, res))
        torch.cuda.synchronize()
    barrier(world)
    step_ms = [ev[i].elapsed_time(ev[i + 1]) for i in range(K)]
    elapsed = sum(step_ms) / 1e3
    launches = _lib.kernel_launches() - launches0
    # per-launch device time of the dominant kernel: the first (up to 3) timed sectors again with
    # per-launch events (which need separate launches: the timed steps are cooperative kernels)
    h.profile(True)
    hc_info = []
    for sidx, _, _ in all_vals[:3]:
        step_device(sidx)
        hc_info.append(h.hit_cache_info())              # the cache the solve built (None: candidate map)
    torch.cuda.synchronize()
    n_mv, ms_mv = h.profile_read(_lib.KERNEL_BLOCK_MATVEC_C64)
    n_hc, ms_hc = h.profile_read(_lib.KERNEL_HC_BLOCK_C64)
    h.profile(False)
    use_hc = n_hc > 0
    if use_hc:
        n_mv, ms_mv = n_hc, ms_hc
    tuning = h.block_tuning(32, _lib.PREC_MIXED, True)
    # algorithmic bytes of the dominant kernel (c64 block map), averaged over the profiled sectors
    mv_bytes = []
    for (sidx, _, _), hc in zip(all_vals[:3], hc_info):
        if use_hc:
            mv_bytes.append(hc_bytes(len(sectors[sidx][1]), hc["hits"], len(amp_a), 32, 8))
        else:
            h.select_sector(sidx, len(sectors[sidx][1]))
            st = h.stats()
            mv_bytes.append(block_bytes(len(sectors[sidx][1]), st["nnz"], len(amp_a), 32, 8))
    bytes_per_launch = float(np.mean(mv_bytes))
    solves_local = K * NU
    elapsed_max = all_max(elapsed, world)
    solves_total = all_sum(solves_local, world)
    value = solves_total / elapsed_max

    # ---------------------------------------------------------------- e2e: public API, host buffers
    def pinned(shape, dtype):
        t = torch.empty(int(np.prod(shape)) * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
        return t, t.numpy().view(dtype).reshape(shape)

    keep_alive = []
    host_inputs = []
    for i in range(K):                                   # this step's inputs in pinned host memory
        src = sectors[order[W + i]][1]
        t, b = pinned(src.shape, np.uint64)
        b[:] = src
        keep_alive.append(t)
        host_inputs.append(b)
    pair_host = []
    for a in (amp_a, amp_b, in_, out, pm):
        t, b = pinned(a.shape, a.dtype)
        b[:] = a
        keep_alive.append(t)
        pair_host.append(b)
    nmax = max(len(b) for b in host_inputs)
    t, vec_host = pinned((NU * NEV * nmax,), np.complex128)
    keep_alive.append(t)
    h2d = [b.nbytes + sum(a.nbytes for a in pair_host) for b in host_inputs]
    barrier(world)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e2e_ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e2e_ev[0].record(stream)
    d2h = []
    for i in range(K):
        h.set_basis(host_inputs[i])
        h.set_scatter_pair(*pair_host)
        nb = len(host_inputs[i])
        vals, vecs, res, info = h.batch_solve(u, NEV, krylovdim=KRYLOV, tol=1e-12, precision=_lib.PREC_MIXED,
                                              want_vectors=True,
                                              out_vecs=vec_host[:NU * NEV * nb].reshape(NU, NEV, nb))
        d2h.append(vals.nbytes + res.nbytes + vecs.nbytes)
    e2e_ev[1].record(stream)
    torch.cuda.synchronize()
    e2e_elapsed = all_max(e2e_ev[0].elapsed_time(e2e_ev[1]) / 1e3, world)
    e2e_value = all_sum(solves_local, world) / e2e_elapsed

    # ---------------------------------------------------------------- plain one-at-a-time FP64 GPU Lanczos
    plain = None
    if rank == 0 and args.plain > 0:
        # the same sectors as the timed steps, args.plain U0 values spread over the grid on each
        h.set_scatter_pair(amp_a, amp_b, in_, out, pm)
        picks = sorted({int(round(j * (NU - 1) / max(args.plain - 1, 1))) for j in range(args.plain)})
        lat, errs = [], []
        os.environ["MOMED_BLOCK"] = "0"          # the plain GPU Lanczos: single-vector Krylov
        for sidx, bvals, _ in all_vals:
            h.select_sector(sidx, len(sectors[sidx][1]))
            h.set_param(float(u[picks[0]]))               # untimed: this sector's index and operator checks
            h.eigsolve(NEV, krylovdim=KRYLOV, tol=1e-12, seed=1, want_vectors=False, precision=_lib.PREC_FP64)
            for j in picks:
                h.set_param(float(u[j]))
                pe = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                torch.cuda.synchronize()
                pe[0].record(stream)
                pv, _, pr, pinfo = h.eigsolve(NEV, krylovdim=KRYLOV, tol=1e-12, seed=1, want_vectors=False,
                                              precision=_lib.PREC_FP64)
                pe[1].record(stream)
                torch.cuda.synchronize()
                lat.append(pe[0].elapsed_time(pe[1]))
                errs.append(float(np.max(np.abs(bvals[j] - pv) / np.maximum(np.abs(pv), 1.0))))
        # the same solves on the sparse method: one matrix per (sector, U0), built inside the timing
        lat_sp = []
        for sidx, bvals, _ in all_vals:
            h.select_sector(sidx, len(sectors[sidx][1]))
            for j in picks:
                h.set_param(float(u[j]))
                pe = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                torch.cuda.synchronize()
                pe[0].record(stream)
                h.build_sparse()
                pv, _, _, _ = h.eigsolve(NEV, krylovdim=KRYLOV, tol=1e-12, seed=1, want_vectors=False,
                                         precision=_lib.PREC_FP64)
                pe[1].record(stream)
                torch.cuda.synchronize()
                lat_sp.append(pe[0].elapsed_time(pe[1]))
                errs.append(float(np.max(np.abs(bvals[j] - pv) / np.maximum(np.abs(pv), 1.0))))
        h.release_sparse()
        os.environ.pop("MOMED_BLOCK", None)
        # the same solves by the library's default FP64 solver (block Lanczos, B = 4 for nev 4)
        lat_bl = []
        for sidx, bvals, _ in all_vals:
            h.select_sector(sidx, len(sectors[sidx][1]))
            for j in picks:
                h.set_param(float(u[j]))
                pe = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                torch.cuda.synchronize()
                pe[0].record(stream)
                pv, _, _, _ = h.eigsolve(NEV, krylovdim=KRYLOV, tol=1e-12, seed=1, want_vectors=False,
                                         precision=_lib.PREC_FP64)
                pe[1].record(stream)
                torch.cuda.synchronize()
                lat_bl.append(pe[0].elapsed_time(pe[1]))
                errs.append(float(np.max(np.abs(bvals[j] - pv) / np.maximum(np.abs(pv), 1.0))))
        h.set_param(1.0)
        plain = {"solves_per_s": 1e3 * len(lat) / sum(lat), "latency_ms_p50": float(np.percentile(lat, 50)),
                 "latency_ms_p99": float(np.percentile(lat, 99)), "solves": len(lat),
                 "sample": f"{len(picks)} U0 values on each of the {len(all_vals)} timed sectors",
                 "max_rel_eig_err_batched_vs_fp64": max(errs),
                 "sparse_method": {"solves_per_s": 1e3 * len(lat_sp) / sum(lat_sp),
                                   "latency_ms_p50": float(np.percentile(lat_sp, 50)),
                                   "note": "the same solves with the matrix built per (sector, U0) inside the timing"},
                 "block_solver": {"solves_per_s": 1e3 * len(lat_bl) / sum(lat_bl),
                                  "latency_ms_p50": float(np.percentile(lat_bl, 50)),
                                  "note": "the same solves by the default FP64 solver (block Lanczos) on the map"},
                 "solver": "single-vector FP64 Lanczos on the map (the reference's Krylov method)"}

    # ---------------------------------------------------------------- the same sweep on the sparse method
    # (each step builds the sector's CSR entries with A and B parts, then the batched solver runs its
    # FP32 maps as a block SpMV over them; reported beside the map-based headline, not as it)
    sparse_batched = None
    if rank == 0 and world == 1 and args.sparse_batch:
        h.set_scatter_pair(amp_a, amp_b, in_, out, pm)

        def step_sparse(sidx):
            h.select_sector(sidx, len(sectors[sidx][1]))
            h.build_sparse()
            return h.batch_solve(u, NEV, krylovdim=KRYLOV, tol=1e-12, precision=_lib.PREC_MIXED)

        step_sparse(order[0])                              # warm-up
        h.profile(True)
        sev = [torch.cuda.Event(enable_timing=True) for _ in range(K + 1)]
        errs = []
        torch.cuda.synchronize()
        sev[0].record(stream)
        for i, (sidx, bvals, _) in enumerate(all_vals):
            sv, _, _, _ = step_sparse(sidx)
            sev[i + 1].record(stream)
            errs.append(float(np.max(np.abs(sv - bvals) / np.maximum(np.abs(bvals), 1.0))))
        torch.cuda.synchronize()
        sms = [sev[i].elapsed_time(sev[i + 1]) for i in range(K)]
        n_bsp, ms_bsp = h.profile_read(_lib.KERNEL_BLOCK_SPMV_C64)
        h.profile(False)
        h.release_sparse()
        sparse_batched = {"solves_per_s": 1e3 * K * NU / sum(sms), "ms_per_step": sum(sms) / K,
                          "block_spmv_launches": n_bsp, "block_spmv_avg_ms": ms_bsp / max(n_bsp, 1),
                          "max_rel_eig_err_vs_map_batched": max(errs),
                          "note": "build of the sector's entries inside each step; same sectors and U0 grid"}

    # ---------------------------------------------------------------- CPU baseline (rank 0, N = 1)
    cpu = None
    eig_vs_oracle = None
    if rank == 0 and world == 1 and not args.no_cpu:
        basis = sectors[order[W]][1]
        nthreads = os.cpu_count() or 1
        dt, ovals, _ = cpu_reference_solve(basis, pair, float(u[0]), nthreads)
        cpu = {"value": 1.0 / dt, "unit": "solves/s", "cores": nthreads, "kind": "port",
               "sample": f"1 full FP64 solve (reference CPU map + Lanczos) of one (sector, U0) pair, "
                         f"{len(basis)} states, U0={u[0]:.3f}"}
        # the batched mixed-precision result of the same (sector, U0) against the FP64 oracle
        bv = np.asarray(all_vals[0][1])[0]
        eig_vs_oracle = {"max_rel_err": float(np.max(np.abs(bv - ovals) / np.abs(ovals))),
                         "per_eigenvalue": [float(v) for v in np.abs(bv - ovals) / np.abs(ovals)],
                         "pair": f"sector {all_vals[0][0]}, U0={u[0]:.3f}, nev {NEV}"}

    serving = None
    if rank == 0 and world == 1 and not args.no_serve and args.serve_requests > 0:
        serving = serve_bench(args, local)

    if rank == 0:
        avg_ms = ms_mv / max(n_mv, 1)
        achieved = bytes_per_launch / (avg_ms * 1e-3) / 1e9
        peaks_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
        peak, peak_src = 6650.0, "fallback"
        if os.path.exists(peaks_path):
            try:
                peak = float(json.load(open(peaks_path))["hbm_gbs"])
                peak_src = "measured"
            except Exception:
                pass
        lat = sorted(step_ms)
        line = {
            "metric": METRIC,
            "value": value, "unit": "solves/s", "n_gpus": world, "steps": K, "warmup": W,
            "ms_per_step": elapsed_max * 1e3 / K, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "c64 matvec / f64 recurrences + f64 Rayleigh-Ritz", "data": "synthetic",
            "config": {"workload": workload_name(),
                       "global_batch": NU * world, "parallelism": f"replicas x{world}",
                       "l2": "inputs larger than L2 (Krylov basis ~1.4 GB per step)"},
            "latency_ms": {"per_batch_p50": float(np.percentile(lat, 50)),
                           "per_batch_p99": float(np.percentile(lat, 99)),
                           "per_solve_p50": float(np.percentile(lat, 50)),
                           "per_solve_p99": float(np.percentile(lat, 99))},
            "plain_gpu_lanczos": plain,
            "speedup_vs_plain": (value / world) / plain["solves_per_s"] if plain else None,
            "speedup_vs_plain_sparse": (value / world) / plain["sparse_method"]["solves_per_s"] if plain else None,
            "sparse_method_batched": sparse_batched,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": MV_DRAM_BYTES_HC if use_hc else MV_DRAM_BYTES,
                         "peak_source": peak_src,
                         "kernel": ("block map c64 x32 over the hit cache (k_block_hc<float, 32>)" if use_hc
                                    else "block matvec c64 x32 (k_block_matvec_v<float, 32>)"),
                         "dram_frac": ((MV_DRAM_BYTES_HC if use_hc else MV_DRAM_BYTES) / (avg_ms * 1e-3) / 1e9 / peak),
                         "note": "algorithmic bytes count one 32-wide x-row gather per hit; x (44 MB) stays in "
                                 "L2, so those gathers are L2 traffic and DRAM moves only the traffic bytes "
                                 "(dram_frac: their rate against the copy peak)",
                         "launches": n_mv, "avg_launch_ms": avg_ms,
                         "algorithmic_bytes_per_launch": bytes_per_launch},
            "cpu_baseline": cpu,
            "eig_err_vs_fp64_oracle": eig_vs_oracle,
            "serving": serving,
            "e2e": {"value": e2e_value, "unit": "solves/s", "h2d_bytes_per_step": int(np.mean(h2d)),
                    "d2h_bytes_per_step": int(np.mean(d2h))},
            "gpu_launches": int(all_sum(launches, world)),
            "clocks": clk.summary(),
            "batching": {"step": "block map + one cooperative launch (projection, update, second pass, scaling)",
                         "block_map_autotune": tuning},
            "hit_cache": ({"hits_per_sector": float(np.mean([c["hits"] for c in hc_info])),
                           "bytes_per_sector": float(np.mean([c["bytes"] for c in hc_info])),
                           "build_ms": float(np.mean([c["build_ms"] for c in hc_info])),
                           "note": "built inside each timed step, at the sector's first map"}
                          if use_hc else None),
            "solver": {"matvecs_per_step": int(np.mean([i["matvecs"] for i in infos])),
                       "fp64_matvecs_per_step": int(np.mean([i["matvecs_fp64"] for i in infos])),
                       "restarts_per_step": float(np.mean([i["restarts"] for i in infos])),
                       "converged_min": int(min(i["converged"] for i in infos)),
                       "max_residual": float(max(float(np.max(r)) for _, _, r in all_vals))},
        }
        print(json.dumps(line), flush=True)
    h.close()
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
