#!/usr/bin/env python
"""SpGEMM benchmark: C = A*A on the R-MAT 2^18 graph (average degree 16,
(a,b,c,d) = (0.57,0.19,0.19,0.05), duplicates removed, values U(0,1]) on one
B200 per process.

One step = one complete product through the engine's C ABI: A given as CSC
and B as CSR, already resident in HBM; symbolic pass, numeric pass and the
sorted CSR of C (row pointers, columns, values) written to device memory.
`value` = GFLOP/s counted as 2 x intermediate products, summed over ranks,
with the time taken as the max over ranks of the summed per-step CUDA-event
times (L2 flushed before every step: the inputs, 63 MB, fit in L2).

Also printed on the same JSON line:
  roofline      the dominant kernel's algorithmic bytes / its CUDA-event time,
                against the measured HBM copy bandwidth;
  pipeline      the same for the whole step;
  e2e           the same metric through spgemm_multiply_host_to with pinned
                host buffers: host->device copy of A and B, the product, and
                the device->host copy of all of C inside the timed region;
  cpu_baseline  the CPU restatement of the reference algorithm (FP32, all
                host threads) on a bounded random sample of C's rows;
  clocks        nvidia-smi samples taken during the timed region.

--impl reference times that CPU restatement alone (the reference has no CPU
multiply of its own and its GPU engine cannot run these inputs: int32
overflow at P > 2^31, src/mm.cu:176-184).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "SpGEMM GFLOP/s + HBM GB/s vs roofline; batched/compensated vs plain at 1e-6"
L2_FLUSH_BYTES = 512 << 20


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--workload", choices=["rmat", "stencil", "stencil-comp", "er", "galerkin",
                                          "batch"],
                   default="rmat")
    p.add_argument("--batch-count", type=int, default=512)
    p.add_argument("--loop-steps", type=int, default=2,
                   help="batch: timed passes of the one-product-per-launch loop")
    p.add_argument("--no-autotune", action="store_true")
    p.add_argument("--scale", type=int, default=18, help="R-MAT scale (default 18)")
    p.add_argument("--grid", type=int, default=96,
                   help="stencil grid side (default 96; smaller grids for profiling)")
    p.add_argument("--e2e-steps", type=int, default=3)
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--cpu-seconds", type=float, default=8.0)
    p.add_argument("--no-configs", action="store_true",
                   help="skip the per-configuration suite of the default line")
    p.add_argument("--tune", default="",
                   help="tuning overrides for the GPU arm, e.g. long_rows=1,long_p=2048")
    return p.parse_args()


# ---------------------------------------------------------------------------
# workloads
# ---------------------------------------------------------------------------

def tune_overrides(args):
    """--tune "k=v,k=v" as a dict of spgemm_tuning fields."""
    out = {}
    for kv in filter(None, args.tune.split(",")):
        k, v = kv.split("=")
        out[k.strip()] = int(v)
    return out


def build_workload(args):
    from spgemm_b200 import workloads as W
    if args.workload == "rmat":
        A = W.rmat(args.scale, 16, 0)
        return {"name": f"rmat{args.scale}_ef16_AxA", "products": [(A, A)], "precision": 0,
                "config": {"workload": f"R-MAT 2^{args.scale} ef16 (0.57,0.19,0.19,0.05) dedup, "
                                       "values U(0,1], C = A*A", "rows": A.rows, "nnz_a": A.nnz}}
    if args.workload in ("stencil", "stencil-comp"):
        g = args.grid
        A = W.stencil27(g, seed=0)
        comp = args.workload == "stencil-comp"
        return {"name": f"stencil{g}_27pt_AxA" + ("_compensated" if comp else ""),
                "products": [(A, A)], "precision": 1 if comp else 0,
                "config": {"workload": f"27-point stencil {g}^3, random sign, |v| log-uniform "
                                       f"[1e-4,1e4], C = A*A, {'compensated' if comp else 'plain'} FP32",
                           "rows": A.rows, "nnz_a": A.nnz}}
    if args.workload == "er":
        A = W.er(4096, 8.0, 0)
        return {"name": "er4096_AxA", "products": [(A, A)], "precision": 0,
                "config": {"workload": "Erdos-Renyi 4096, 8/row, U[-1,1], C = A*A",
                           "rows": A.rows, "nnz_a": A.nnz}}
    if args.workload == "galerkin":
        A = W.stencil27(64, values="laplace")
        P = W.prolongator(64)
        return {"name": "galerkin64_PtAP", "products": [(A, P), ("PT", "AP")], "precision": 1,
                "A": A, "P": P,
                "config": {"workload": "Galerkin P^T (A P), A 27-pt 64^3 (26/-1), P 2x2x2 "
                                       "aggregates, compensated FP32", "rows": A.rows}}
    raise ValueError(args.workload)


def product_stats(A, B):
    """Per-row P_i, nnz(A(i,:)), the column span of the row's products, and the
    B bytes touched (for the roofline)."""
    deg_b = np.diff(B.rowptr).astype(np.int64)
    rows_of = np.repeat(np.arange(A.rows), np.diff(A.rowptr))
    p_i = np.zeros(A.rows, np.int64)
    np.add.at(p_i, rows_of, deg_b[A.col])
    touched_k = np.zeros(B.rows, bool)
    touched_k[A.col] = True
    b_touched = 4 * (B.rows + 1) + 8 * int(deg_b[touched_k].sum())
    nonempty = deg_b > 0
    first = np.full(B.rows, np.iinfo(np.int64).max)
    last = np.full(B.rows, -1)
    first[nonempty] = B.col[B.rowptr[:-1][nonempty]]
    last[nonempty] = B.col[B.rowptr[1:][nonempty] - 1]
    lo = np.full(A.rows, np.iinfo(np.int64).max)
    hi = np.full(A.rows, -1)
    np.minimum.at(lo, rows_of, first[A.col])
    np.maximum.at(hi, rows_of, last[A.col])
    span = np.where(p_i > 0, hi + 1 - (lo & ~31), 0)
    return p_i, np.diff(A.rowptr).astype(np.int64), b_touched, span


# Mirrors of the engine's default bin rules (kernels.cuh), used only to
# attribute algorithmic bytes to the kernel that processed each row.
LONG_P, WARP_CAP, WARP_TMAX, MID_COLS, LONG_O, MID_O = 4096, 2048, 256, 1 << 18, 4096, 256
ESC_P = {32: 256, 64: 512, 128: 1024, 256: 2048, 512: 4096}  # products of a sorted row, by block size
# output capacities of the whole-row kernel's two block sizes (engine.cu:
# (shared-memory budget - per-warp scratch - directory) / 4 bytes)
ROWS_CAP_512 = (111 * 1024 - 16 * 384 - 8193 * 8) // 4
ROWS_CAP_1024 = (225 * 1024 - 32 * 384 - 8193 * 8) // 4


def row_kernel(p, cap, span):
    """Kernel of each row's first pass, as the profile names it. Warp-table
    rows are put down as hashed: the engine sorts those of a neighbourhood
    whose products hardly share columns, which only a sample of A's entries
    tells."""
    lg = np.ceil(np.log2(np.maximum(cap + cap // 4 + 1, 1))).astype(np.int64)
    bin_ = np.clip(lg, 6, int(np.log2(WARP_TMAX))) - 6
    name = np.array([f"k_fused_warp<{b}>" for b in range(5)], dtype=object)[bin_]
    name[span <= 4096 - 31] = "k_fused_bits"
    name[p <= 32] = "k_fused_tiny"
    wide = cap > WARP_CAP
    below = 0
    for nt, most in ESC_P.items():
        name[wide & (p > below) & (p <= most)] = f"k_fused_esc<{nt}>"
        below = most
    name[(p > LONG_P) | (p <= 0)] = ""
    return name


def kernel_rows(name, p_i, o_i, span, n):
    """Rows processed by an engine kernel (mask), and whether it writes C."""
    cap = np.minimum(np.minimum(p_i, n), span)
    long_rows = p_i > LONG_P
    if name == "k_sym_long":
        return long_rows, False
    # whole long rows (default long_rows=2): up to ROWS_CAP_512 outputs in
    # 512-thread blocks, up to ROWS_CAP_1024 in 1024-thread blocks, column
    # slices (k_num_long) above
    if name == "k_num_rows<512>":
        return long_rows & (o_i > 0) & (o_i <= ROWS_CAP_512) & (span <= (1 << 18)), True
    if name == "k_num_rows<1024>":
        return long_rows & (o_i > ROWS_CAP_512) & (o_i <= ROWS_CAP_1024) & (span <= (1 << 18)), True
    if name == "k_num_long":
        return long_rows & (o_i > LONG_O) & ((o_i > ROWS_CAP_1024) | (span > (1 << 18))), True
    if name == "k_num_mid":
        return long_rows & (o_i > MID_O) & (o_i <= LONG_O) & (span <= MID_COLS), True
    if name.startswith("k_fused_"):
        # one column a slot, or both forms of the table in one launch
        name = name.replace("warp+cols", "warp").replace("k_fused_cols", "k_fused_warp")
        sel = row_kernel(p_i, cap, span) == name
        return (sel, True) if sel.any() else (None, False)
    return None, False


def algorithmic_bytes(rows_sel, p_i, a_len, o_i, b_touched, p_total, with_c=True):
    """The bytes of A + B rows touched + 8 bytes per partial + C (the
    roofline's algorithmic bytes) restricted to the selected rows; B's share
    is apportioned by partial products."""
    p = int(p_i[rows_sel].sum())
    a = 4 * (int(rows_sel.sum()) + 1) + 8 * int(a_len[rows_sel].sum())
    b = int(round(b_touched * (p / max(p_total, 1))))
    c = (4 * (int(rows_sel.sum()) + 1) + 8 * int(o_i[rows_sel].sum())) if with_c else 4 * int(rows_sel.sum())
    return a + b + 8 * p + c


# ---------------------------------------------------------------------------
# measurement helpers
# ---------------------------------------------------------------------------

class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = Path(os.environ.get("TMPDIR", "/tmp")) / f"spgemm_clocks_{os.getpid()}.csv"

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if not self.proc:
            return None
        time.sleep(0.3)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], 0.0, set()
        for line in self.path.read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for name, v in zip(["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
                                "sw_power_cap"], f[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        try:
            self.path.unlink()
        except OSError:
            pass
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


# ncu summaries (profiles/) of the dominant kernel's DRAM traffic per launch,
# by (workload, kernel): the roofline's "traffic" field.
TRAFFIC_PROFILES = {("rmat18", "k_num_long"): ROOT / "profiles" / "k_num_long_rmat17_traffic.md"}


def profiled_traffic(workload, kernel):
    p = TRAFFIC_PROFILES.get((workload, kernel))
    if p is None or not p.exists():
        return None
    for line in p.read_text().splitlines():
        if line.startswith("traffic_bytes_per_launch:"):
            return int(line.split(":", 1)[1].strip())
    return None


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def cpu_baseline(A, B, target_seconds, seed=0):
    """FP32 CPU restatement of the reference algorithm (oracle mode 1), all
    host threads, on a random sample of rows sized for ~target_seconds."""
    import oracle
    a = A.to_csc()
    threads = os.cpu_count() or 1
    p_i = product_stats(A, B)[0]
    rng = np.random.default_rng(seed)
    order = rng.permutation(A.rows).astype(np.int32)
    csum = np.cumsum(p_i[order])

    def run(target_p):
        k = int(np.searchsorted(csum, target_p)) + 1
        rows = np.sort(order[:min(k, A.rows)])
        t0 = time.perf_counter()
        r = oracle.spgemm(A.rows, B.cols, a.colptr, a.rowidx, a.val, B.rowptr, B.col, B.val,
                          rows=rows, mode=1, threads=threads)
        dt = time.perf_counter() - t0
        return dt, r["products"], len(rows)

    dt, prods, _ = run(min(2e7, csum[-1]))
    rate = prods / max(dt, 1e-9)
    target = min(rate * target_seconds, float(csum[-1]))
    dt, prods, nrows = run(target)
    return {"value": 2.0 * prods / dt / 1e9, "unit": "GFLOP/s", "cores": threads, "kind": "port",
            "sample": f"{nrows} random rows of C ({prods} of {int(csum[-1])} products, "
                      f"{100.0 * prods / csum[-1]:.1f}%), {dt:.2f} s"}, (dt, prods, nrows)


# ---------------------------------------------------------------------------
# reference arm
# ---------------------------------------------------------------------------

def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    wl = build_workload(args)
    A, B = wl["products"][0]
    if isinstance(A, str):
        A, B = wl["A"], wl["P"]
    for _ in range(args.warmup):
        cpu_baseline(A, B, 1.0)
    vals = []
    last = None
    for k in range(args.steps):
        cb, last = cpu_baseline(A, B, 4.0, seed=k)
        vals.append(cb["value"])
    value = float(np.mean(vals))
    dt, prods, nrows = last
    line = {"metric": METRIC, "impl": "reference", "value": value, "unit": "GFLOP/s",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": dt * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded generator)",
            "config": wl["config"],
            "cpu_baseline": {"value": value, "unit": "GFLOP/s", "cores": os.cpu_count(),
                             "kind": "port",
                             "sample": f"per step: random rows of C sized for ~4 s "
                                       f"(last: {nrows} rows, {prods} products)"},
            "e2e": {"value": value, "unit": "GFLOP/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0},
            "note": "the reference has no CPU multiply; this is the oracle's FP32 restatement "
                    "of its algorithm (src/mm.cu initGEMM/binGEMM/mergeGEMM), all host threads"}
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# batch workload: 512 independent products, one captured graph per step
# ---------------------------------------------------------------------------

def _batch_item(spec):
    from spgemm_b200 import workloads as W
    it = W.batch_item(*spec)
    return it.A, it.B


def build_batch(count, seed=1000):
    """The 512-product batch (n log-uniform [1k, 200k], Poisson(lam) nnz/row
    with lam ~ U[4, 32], half ER / half R-MAT, values U[-1, 1], seed + i per
    instance), generated on all host cores."""
    from spgemm_b200 import workloads as W
    specs = W.batch_specs(count, seed)
    workers = min(os.cpu_count() or 1, 32)
    if workers > 1:
        import multiprocessing as mp
        with mp.get_context("spawn").Pool(workers) as pool:
            pairs = pool.map(_batch_item, specs, chunksize=1)
    else:
        pairs = [_batch_item(sp) for sp in specs]
    return specs, pairs


def batch_products(pairs):
    """Total intermediate products and the roofline's algorithmic bytes
    (A + B rows touched + partials + C is added after the run)."""
    P, ab = 0, 0
    for A, B in pairs:
        deg_b = np.diff(B.rowptr.astype(np.int64))
        p = int(deg_b[A.col].sum())
        P += p
        touched = np.zeros(B.rows, bool)
        touched[A.col] = True
        ab += 4 * (A.rows + 1) + 8 * A.nnz + 4 * (B.rows + 1) + 8 * int(deg_b[touched].sum()) + 8 * p
    return P, ab


def measure_batch(args, dev, stream, pairs, steps, warmup, loop_steps, rank=0, dist=None,
                  smi_id="0"):
    """The batched form's measurement: operands uploaded into one device
    arena per array kind, the batch planned (autotuned unless --no-autotune),
    `steps` graph replays timed with CUDA events (L2 flushed before each),
    the kernel split of one step, and the plain loop (one spgemm_multiply per
    product) timed `loop_steps` times. Returns a dict; its handle "hb" stays
    open for the caller."""
    import torch
    import spgemm_b200 as sg
    from spgemm_b200 import autotune
    P, alg_in = batch_products(pairs)

    # operands in one device arena per array kind (inputs stay resident)
    def arena(parts, dt):
        sizes = [len(x) for x in parts]
        host = torch.from_numpy(np.concatenate([np.asarray(x) for x in parts]).astype(
            np.int32 if dt == torch.int32 else np.float32))
        return host, np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    kinds = {}
    for name, getter, dt in [("a_ptr", lambda A, B: A.rowptr, torch.int32),
                             ("a_col", lambda A, B: A.col, torch.int32),
                             ("a_val", lambda A, B: A.val, torch.float32),
                             ("b_ptr", lambda A, B: B.rowptr, torch.int32),
                             ("b_col", lambda A, B: B.col, torch.int32),
                             ("b_val", lambda A, B: B.val, torch.float32)]:
        host, off = arena([getter(A, B) for A, B in pairs], dt)
        pinned = host.pin_memory()
        devt = torch.empty(max(host.numel(), 1), dtype=dt, device=dev)
        devt[:host.numel()].copy_(pinned)
        kinds[name] = (pinned, devt, off)
    esz = 4

    def addr(name, i):
        return kinds[name][1].data_ptr() + int(kinds[name][2][i]) * esz
    A_list = [sg.device_cm(addr("a_ptr", i), addr("a_col", i), addr("a_val", i), A.nnz, A.rows,
                           A.cols, sg.ROW_MAJOR) for i, (A, B) in enumerate(pairs)]
    B_list = [sg.device_cm(addr("b_ptr", i), addr("b_col", i), addr("b_val", i), B.nnz, B.rows,
                           B.cols, sg.ROW_MAJOR) for i, (A, B) in enumerate(pairs)]
    torch.cuda.synchronize()

    hb = sg.Handle(sg.PLAIN)
    if tune_overrides(args):
        hb.set_tuning(**tune_overrides(args))
    hb.set_stream(stream.cuda_stream)
    if args.no_autotune:
        nnz_total = hb.batch_plan(A_list, B_list)
        tune = {"tuning": None, "tried": 0, "cached": False}
    else:
        tune = autotune.tune_batch(hb, A_list, B_list, torch.cuda.get_device_name(dev), cache=None)
        nnz_total = hb.stats()["nnz_c"]
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device=dev)
    for _ in range(max(warmup, 0)):
        hb.batch_execute(graph=True)
    torch.cuda.synchronize()
    launches0 = hb.stats()["kernel_launches"]
    if dist:
        dist.barrier()
    sampler = ClockSampler(smi_id) if rank == 0 else None
    if sampler:
        sampler.start()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(steps)]
    for k in range(steps):
        flush.zero_()
        ev[k][0].record(stream)
        hb.batch_execute(graph=True)
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    clocks = sampler.stop() if sampler else None
    step_ms = [a.elapsed_time(b) for a, b in ev]
    total_ms = float(sum(step_ms))
    launches = hb.stats()["kernel_launches"] - launches0
    if dist:
        t = torch.tensor([total_ms], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())

    # kernel split of one step (direct launches with timing events; untimed)
    hb.reset_kernel_times()
    hb.set_profiling(True)
    hb.batch_execute(graph=False)
    hb.set_profiling(False)
    ktimes = sorted(hb.kernel_times().items(), key=lambda kv: -kv[1][0])

    # plain path: one spgemm_multiply per product (same operands, same stream)
    hp = sg.Handle(sg.PLAIN)
    hp.set_stream(stream.cuda_stream)
    for A_cm, B_cm in zip(A_list, B_list):  # warm-up (allocations)
        hp.multiply(A_cm, B_cm)
    torch.cuda.synchronize()
    loop_ms = []
    for _ in range(max(loop_steps, 1)):
        s0, s1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        flush.zero_()
        s0.record(stream)
        for A_cm, B_cm in zip(A_list, B_list):
            hp.multiply(A_cm, B_cm)
        s1.record(stream)
        torch.cuda.synchronize()
        loop_ms.append(s0.elapsed_time(s1))
    loop_step = float(np.median(loop_ms))
    hp.close()
    del flush
    ro, no = hb.batch_offsets()
    return {"hb": hb, "P": P, "alg_in": alg_in, "kinds": kinds, "nnz_total": nnz_total,
            "tune": tune, "step_ms": step_ms, "total_ms": total_ms, "clocks": clocks,
            "launches": launches, "ktimes": ktimes, "loop_step": loop_step, "ro": ro, "no": no}


def run_batch(args):
    """Batched form: every step recomputes all products from the operands in
    HBM by one replay of the batch's CUDA graph (pack, analysis, fused and
    long-row passes of the packed block-diagonal product, per-product row
    pointers), tuned by spgemm_b200.autotune. Compared with the plain path:
    the same products one spgemm_multiply call each."""
    specs, pairs = build_batch(args.batch_count)  # before any CUDA use (spawned workers)
    import torch
    import spgemm_b200 as sg
    local = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    stream = torch.cuda.current_stream()
    vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
    smi_id = vis.split(",")[local].strip() if vis else str(local)
    res = measure_batch(args, dev, stream, pairs, args.steps, args.warmup, args.loop_steps,
                        rank, dist, smi_id)
    hb, P, alg_in, kinds = res["hb"], res["P"], res["alg_in"], res["kinds"]
    nnz_total, tune, step_ms, total_ms = res["nnz_total"], res["tune"], res["step_ms"], res["total_ms"]
    clocks, launches, ktimes, loop_step = res["clocks"], res["launches"], res["ktimes"], res["loop_step"]
    ro = res["ro"]
    value = 2.0 * P * args.steps * world / (total_ms / 1e3) / 1e9
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device=dev)

    # e2e: operand arrays host->device (pinned), the batch, all of C device->host
    ro, no = hb.batch_offsets()
    out_rp = torch.empty(int(ro[-1]) + len(pairs), dtype=torch.int32).pin_memory()
    out_col = torch.empty(max(int(nnz_total), 1), dtype=torch.int32).pin_memory()
    out_val = torch.empty(max(int(nnz_total), 1), dtype=torch.float32).pin_memory()
    h2d = sum(v[0].numel() * 4 for v in kinds.values())
    d2h = (out_rp.numel() + 2 * int(nnz_total)) * 4
    e_ms = []
    for _ in range(max(args.e2e_steps, 1) + 1):
        s0, s1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s0.record(stream)
        for pinned, devt, _ in kinds.values():
            devt[:pinned.numel()].copy_(pinned, non_blocking=True)
        hb.batch_execute(graph=True)
        hb.batch_copy_all(out_rp.data_ptr(), out_col.data_ptr(), out_val.data_ptr())
        s1.record(stream)
        torch.cuda.synchronize()
        e_ms.append(s0.elapsed_time(s1))
    e_ms = e_ms[1:]  # the first pass is a warm-up
    e2e = {"value": 2.0 * P / (float(np.mean(e_ms)) / 1e3) / 1e9, "unit": "GFLOP/s",
           "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
           "ms_per_step": float(np.mean(e_ms))}

    peak, peak_kind = measured_peaks()
    alg = alg_in + 4 * (int(ro[-1]) + len(pairs)) + 8 * int(nnz_total)
    step_s = total_ms / args.steps / 1e3
    roof = {"bound": "hbm", "kernel": "batch graph (whole step)", "achieved": alg / step_s / 1e9,
            "peak": peak, "unit": "GB/s", "frac": alg / step_s / 1e9 / peak, "traffic": None,
            "algorithmic_bytes_per_launch": alg, "avg_launch_ms": step_s * 1e3,
            "peak_kind": peak_kind}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        import oracle
        threads = os.cpu_count() or 1
        rng = np.random.default_rng(0)
        t0 = time.perf_counter()
        prods, used = 0, 0
        for i in rng.permutation(len(pairs)):
            A, B = pairs[i]
            a = A.to_csc()
            r = oracle.spgemm(A.rows, B.cols, a.colptr, a.rowidx, a.val, B.rowptr, B.col, B.val,
                              mode=1, threads=threads)
            prods += r["products"]
            used += 1
            if time.perf_counter() - t0 > args.cpu_seconds:
                break
        dt = time.perf_counter() - t0
        cpu = {"value": 2.0 * prods / dt / 1e9, "unit": "GFLOP/s", "cores": threads,
               "kind": "port", "sample": f"{used} random products of the batch "
                                         f"({prods} of {P} products), {dt:.2f} s"}

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": "GFLOP/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic (seeded generator)",
                "config": {"workload": f"batch of {len(pairs)} independent C_i = A_i*B_i: n_i "
                                       "log-uniform [1k, 200k], Poisson(lam_i) nnz/row, lam_i ~ "
                                       "U[4, 32], half ER / half R-MAT, values U[-1, 1]",
                           "intermediate_products": P, "nnz_c": int(nnz_total),
                           "rows": int(ro[-1]), "nnz_a": int(sum(A.nnz for A, _ in pairs)),
                           "l2": "flushed before every step (512 MiB write); operands exceed L2",
                           "parallelism": f"replicas x{world}"},
                "batched_vs_plain_loop": {"plain_loop_ms": loop_step,
                                          "batched_ms": total_ms / args.steps,
                                          "speedup": loop_step / (total_ms / args.steps),
                                          "plain_loop_gflops": 2.0 * P / (loop_step / 1e3) / 1e9},
                "autotune": {k: tune[k] for k in ("tuning", "tried", "cached") if k in tune},
                "roofline": roof, "cpu_baseline": cpu, "e2e": e2e, "clocks": clocks,
                "gpu_launches": launches,
                "kernel_ms_per_step": {k: v[0] for k, v in ktimes[:12]},
                "step_ms": step_ms}
        print(json.dumps(line), flush=True)
    hb.close()
    if dist:
        dist.destroy_process_group()
    return 0


# ---------------------------------------------------------------------------
# configuration suite: every configuration of the benchmark, one line
# ---------------------------------------------------------------------------

def _csr64(M, absval=False):
    import warnings
    import torch
    warnings.filterwarnings("ignore", message="Sparse")
    v = np.asarray(M.val, np.float64)
    return torch.sparse_csr_tensor(
        torch.from_numpy(np.asarray(M.rowptr, np.int64)),
        torch.from_numpy(np.asarray(M.col, np.int64)),
        torch.from_numpy(np.abs(v) if absval else v), size=(M.rows, M.cols)).cuda()


def _sorted_entries(C, rows, ncols):
    import torch
    crow, col, val = C.crow_indices(), C.col_indices(), C.values()
    r = torch.repeat_interleave(torch.arange(rows, device=col.device), crow.diff())
    key = r * ncols + col
    order = torch.argsort(key)
    return key[order], val[order]


def fp64_product(A, B):
    """C = A*B in FP64 on the GPU by torch's sparse CSR product (cuSPARSE): an
    independent checker for the error report, not the engine. Returns the
    sorted keys (row * n + col) of C's entries, their FP64 values, and the
    keys and values of |A|*|B| (sum of |p| per entry)."""
    k, v = _sorted_entries(_csr64(A) @ _csr64(B), A.rows, B.cols)
    ka, va = _sorted_entries(_csr64(A, True) @ _csr64(B, True), A.rows, B.cols)
    return k, v, ka, va


def fp64_chain(Pt, A, Pm):
    """P^T (A P) in FP64 on the GPU (torch / cuSPARSE), as fp64_product."""
    k, v = _sorted_entries(_csr64(Pt) @ (_csr64(A) @ _csr64(Pm)), Pt.rows, Pm.cols)
    ka, va = _sorted_entries(_csr64(Pt, True) @ (_csr64(A, True) @ _csr64(Pm, True)), Pt.rows,
                             Pm.cols)
    return k, v, ka, va


def rel_error_vs(ref, key, val):
    """Errors of the engine's entries (key, val) against an FP64 product
    `ref` = (keys, values, |p|-sum keys, |p|-sum values): max |v - c| / |c|
    over entries with c != 0, the condition sum|p| / |c| of that entry, and
    max |v - c| / sum|p| (the quantity the FP32 summation bound
    gamma_n * sum|p| limits). Entries the FP64 product does not store count
    as c = 0."""
    import torch
    k64, v64, ka, va = ref

    def at(keys, vals):
        if keys.numel() == 0:
            return torch.zeros_like(val, dtype=torch.float64)
        pos = torch.searchsorted(keys, key).clamp(max=keys.numel() - 1)
        return torch.where(keys[pos] == key, vals[pos], torch.zeros_like(vals[pos]))
    c, absum = at(k64, v64), at(ka, va)
    err = (val.double() - c).abs()
    nz = c != 0
    out = {"zero_entries": int((~nz).sum())}
    if bool(nz.any()):
        rel = torch.where(nz, err / c.abs().clamp(min=1e-300), torch.zeros_like(err))
        w = int(torch.argmax(rel))
        out.update(max_rel=float(rel[w]), worst_cond=float(absum[w] / c[w].abs()))
    else:
        out.update(max_rel=0.0, worst_cond=0.0)
    pos = absum > 0
    out["max_err_over_abssum"] = float((err[pos] / absum[pos]).max()) if bool(pos.any()) else 0.0
    return out


def sampled_row_error(A, B, rp, col, val, nrows=2048, heavy=32):
    """Relative error of C's rows for a sample (nrows random rows and the
    `heavy` rows with the most products) against the FP64 product of those
    rows of A with B (fp64_product)."""
    import torch
    from spgemm_b200 import workloads as W
    p_i = product_stats(A, B)[0]
    rng = np.random.default_rng(0)
    rows = np.unique(np.concatenate([rng.choice(A.rows, min(nrows, A.rows), replace=False),
                                     np.argsort(p_i)[-heavy:]])).astype(np.int64)
    arp = A.rowptr.astype(np.int64)
    lens = arp[rows + 1] - arp[rows]
    sel = np.concatenate([np.arange(arp[i], arp[i + 1]) for i in rows])
    Asub = W.Csr(len(rows), A.cols, np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
                 A.col[sel], A.val[sel])
    ref = fp64_product(Asub, B)
    rp_h = rp.cpu().numpy().astype(np.int64)
    clen = rp_h[rows + 1] - rp_h[rows]
    pos = torch.from_numpy(np.concatenate([np.arange(rp_h[i], rp_h[i + 1]) for i in rows])).cuda()
    sub_row = torch.from_numpy(np.repeat(np.arange(len(rows), dtype=np.int64), clen)).cuda()
    key = sub_row * B.cols + col[pos].long()
    err = rel_error_vs(ref, key, val[pos])
    err["rows_checked"] = int(len(rows))
    return err


def engine_keys(rp, col, n):
    import torch
    rows = torch.repeat_interleave(torch.arange(rp.numel() - 1, device=col.device),
                                   rp.long().diff())
    return rows * n + col.long()


class DeviceProduct:
    """One product through the C ABI on device-resident operands (A as CSC,
    B as CSR), output into preallocated device arrays."""

    def __init__(self, sg, torch, dev, stream, A, B, precision, tune):
        up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype=t)
        Ac = A.to_csc()
        self.keep = [up(Ac.colptr, torch.int32), up(Ac.rowidx, torch.int32), up(Ac.val, torch.float32),
                     up(B.rowptr, torch.int32), up(B.col, torch.int32), up(B.val, torch.float32)]
        k = self.keep
        self.A = sg.device_cm(k[0].data_ptr(), k[1].data_ptr(), k[2].data_ptr(), A.nnz, A.rows,
                              A.cols, sg.COL_MAJOR)
        self.B = sg.device_cm(k[3].data_ptr(), k[4].data_ptr(), k[5].data_ptr(), B.nnz, B.rows,
                              B.cols, sg.ROW_MAJOR)
        self.h = sg.Handle(precision)
        if tune:
            self.h.set_tuning(**tune)
        self.h.set_stream(stream.cuda_stream)
        self.rows, self.torch, self.dev, self.cap = A.rows, torch, dev, -1

    def step(self):
        t = self.torch
        nnz = self.h.symbolic(self.A, self.B)
        if self.cap < nnz:
            self.rp = t.empty(self.rows + 1, dtype=t.int32, device=self.dev)
            self.col = t.empty(max(nnz, 1), dtype=t.int32, device=self.dev)
            self.val = t.empty(max(nnz, 1), dtype=t.float32, device=self.dev)
            self.cap = nnz
        self.nnz = nnz
        self.h.numeric(self.rp.data_ptr(), self.col.data_ptr(), self.val.data_ptr())

    def close(self):
        self.h.close()


def timed(torch, stream, fn, steps, warmup, smi_id):
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    sampler = ClockSampler(smi_id)
    sampler.start()
    ms = []
    for _ in range(steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        flush.zero_()
        a.record(stream)
        fn()
        b.record(stream)
        torch.cuda.synchronize()
        ms.append(a.elapsed_time(b))
    return float(np.mean(ms)), sampler.stop()


def run_suite(args, dev, stream, smi_id):
    """ER 4096, stencil 96^3 (plain and compensated), Galerkin 64^3 (P^T A P,
    compensated) and the 512-product batch, each: ms per step (L2 flushed
    before every step), GFLOP/s (2 x intermediate products), algorithmic
    bytes and their fraction of the measured HBM bandwidth, the maximum
    relative error against an FP64 product (torch/cuSPARSE on the GPU), and
    the clocks seen while timing."""
    import torch
    import spgemm_b200 as sg
    from spgemm_b200 import workloads as W
    peak, peak_kind = measured_peaks()
    tune = tune_overrides(args)
    out = {}

    def prod_bytes(A, B, nnz_c):
        p_i, a_len, b_touched, _ = product_stats(A, B)
        o = np.zeros(A.rows, np.int64)
        rows = np.ones(A.rows, bool)
        base = algorithmic_bytes(rows, p_i, a_len, o, b_touched, int(p_i.sum()), with_c=False)
        return int(p_i.sum()), base - 4 * A.rows + 4 * (A.rows + 1) + 8 * int(nnz_c)

    def single(name, A, B, precision, steps, desc):
        pr = DeviceProduct(sg, torch, dev, stream, A, B, precision, tune)
        ms, clocks = timed(torch, stream, pr.step, steps, 3, smi_id)
        torch.cuda.synchronize()
        P, alg = prod_bytes(A, B, pr.nnz)
        try:
            ref = fp64_product(A, B)
            err = rel_error_vs(ref, engine_keys(pr.rp, pr.col[:pr.nnz], B.cols), pr.val[:pr.nnz])
            del ref
        except Exception as e:  # the checker is optional; the measurement stands
            err = {"unavailable": str(e)[:200]}
        out[name] = {"workload": desc, "precision": "compensated" if precision else "plain",
                     "ms_per_step": ms, "gflops": 2.0 * P / (ms / 1e3) / 1e9,
                     "intermediate_products": P, "nnz_c": int(pr.nnz),
                     "algorithmic_bytes": alg, "gbs": alg / (ms / 1e3) / 1e9,
                     "frac": alg / (ms / 1e3) / 1e9 / peak, "peak_kind": peak_kind,
                     "max_rel_err_vs_fp64": err, "clocks": clocks}
        pr.close()
        torch.cuda.empty_cache()

    A = W.er(4096, 8.0, 0)
    single("er4096", A, A, sg.PLAIN, 50, "ER 4096 x 4096, 8/row, U[-1,1], C = A*A (launch-bound)")
    A = W.stencil27(96, seed=0)
    desc = "27-pt stencil 96^3, random sign, |v| log-uniform [1e-4, 1e4], C = A*A"
    single("stencil96_plain", A, A, sg.PLAIN, 5, desc)
    single("stencil96_compensated", A, A, sg.COMPENSATED, 5, desc)
    del A

    # Galerkin P^T (A P): two chained products, compensated
    A = W.stencil27(64, values="laplace")
    Pm = W.prolongator(64)
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype=t)
    Ac = A.to_csc()
    k = [up(Ac.colptr, torch.int32), up(Ac.rowidx, torch.int32), up(Ac.val, torch.float32),
         up(Pm.rowptr, torch.int32), up(Pm.col, torch.int32), up(Pm.val, torch.float32)]
    A_cm = sg.device_cm(k[0].data_ptr(), k[1].data_ptr(), k[2].data_ptr(), A.nnz, A.rows, A.cols, sg.COL_MAJOR)
    P_cm = sg.device_cm(k[3].data_ptr(), k[4].data_ptr(), k[5].data_ptr(), Pm.nnz, Pm.rows, Pm.cols, sg.ROW_MAJOR)
    PT_cm = sg.device_cm(k[3].data_ptr(), k[4].data_ptr(), k[5].data_ptr(), Pm.nnz, Pm.cols, Pm.rows, sg.COL_MAJOR)
    h1, h2 = sg.Handle(sg.COMPENSATED), sg.Handle(sg.COMPENSATED)
    for h in (h1, h2):
        if tune:
            h.set_tuning(**tune)
        h.set_stream(stream.cuda_stream)
    res = {}

    def chain():
        res["ap"] = h1.multiply(A_cm, P_cm)
        res["c"] = h2.multiply(PT_cm, res["ap"])
    ms, clocks = timed(torch, stream, chain, 10, 3, smi_id)
    P1, P2 = h1.stats()["intermediate_products"], h2.stats()["intermediate_products"]
    nnz_ap = h1.stats()["nnz_c"]
    Pt = Pm.transpose()
    # algorithmic bytes of both products: A*P, then P^T*(AP) (every row of AP touched)
    alg = prod_bytes(A, Pm, nnz_ap)[1]
    # check pass (untimed): the second product once more into caller buffers
    nnz_c = h2.symbolic(PT_cm, res["ap"])
    rp = torch.empty(Pt.rows + 1, dtype=torch.int32, device=dev)
    col = torch.empty(max(nnz_c, 1), dtype=torch.int32, device=dev)
    val = torch.empty(max(nnz_c, 1), dtype=torch.float32, device=dev)
    h2.numeric(rp.data_ptr(), col.data_ptr(), val.data_ptr())
    torch.cuda.synchronize()
    alg += (4 * (Pt.rows + 1) + 8 * Pt.nnz + 4 * (A.rows + 1) + 8 * nnz_ap + 8 * P2 +
            4 * (Pt.rows + 1) + 8 * nnz_c)
    try:
        err = rel_error_vs(fp64_chain(Pt, A, Pm), engine_keys(rp, col[:nnz_c], Pm.cols),
                           val[:nnz_c])
    except Exception as e:
        err = {"unavailable": str(e)[:200]}
    out["galerkin64"] = {"workload": "Galerkin P^T (A P), A 27-pt 64^3 (26/-1), P 2x2x2 aggregates",
                         "precision": "compensated", "ms_per_step": ms,
                         "gflops": 2.0 * (P1 + P2) / (ms / 1e3) / 1e9,
                         "intermediate_products": P1 + P2, "nnz_c": int(nnz_c),
                         "algorithmic_bytes": alg, "gbs": alg / (ms / 1e3) / 1e9,
                         "frac": alg / (ms / 1e3) / 1e9 / peak, "peak_kind": peak_kind,
                         "max_rel_err_vs_fp64": err, "clocks": clocks}
    h1.close()
    h2.close()
    del k, rp, col, val
    torch.cuda.empty_cache()

    # the 512-product batch: one graph replay per step against the plain loop
    _, pairs = build_batch(args.batch_count)
    res = measure_batch(args, dev, stream, pairs, 3, 3, 1, 0, None, smi_id)
    hb = res["hb"]
    ms = res["total_ms"] / 3
    alg = res["alg_in"] + 4 * (int(res["ro"][-1]) + len(pairs)) + 8 * int(res["nnz_total"])
    sizes = [int(np.diff(B.rowptr.astype(np.int64))[A.col].sum()) for A, B in pairs]
    sample = sorted(set(np.random.default_rng(3).choice(len(pairs), 7, replace=False).tolist())
                    | {int(np.argmax(sizes))})
    errs = []
    try:
        for i in sample:
            A, B = pairs[i]
            Cb = hb.batch_copy_result(i)
            ref = fp64_product(A, B)
            rows = np.repeat(np.arange(Cb.rows, dtype=np.int64), np.diff(Cb.rowptr.astype(np.int64)))
            key = torch.from_numpy(rows * B.cols + Cb.col.astype(np.int64)).cuda()
            errs.append(rel_error_vs(ref, key, torch.from_numpy(Cb.val).cuda()))
        err = dict(max(errs, key=lambda e: e["max_rel"]))
        err["max_err_over_abssum"] = max(e["max_err_over_abssum"] for e in errs)
        err["products_checked"] = len(sample)
    except Exception as e:
        err = {"unavailable": str(e)[:200]}
    out["batch512"] = {"workload": f"batch of {len(pairs)} C_i = A_i*B_i (n_i log-uniform "
                                   "[1k, 200k], Poisson(lam_i) nnz/row, lam_i ~ U[4, 32], half ER "
                                   "/ half R-MAT), one CUDA-graph replay per step",
                       "precision": "plain", "ms_per_step": ms,
                       "gflops": 2.0 * res["P"] / (ms / 1e3) / 1e9,
                       "intermediate_products": res["P"], "nnz_c": int(res["nnz_total"]),
                       "algorithmic_bytes": alg, "gbs": alg / (ms / 1e3) / 1e9,
                       "frac": alg / (ms / 1e3) / 1e9 / peak, "peak_kind": peak_kind,
                       "plain_loop_ms": res["loop_step"],
                       "speedup_vs_plain_loop": res["loop_step"] / ms,
                       "autotune": {k: res["tune"][k] for k in ("tuning", "tried") if k in res["tune"]},
                       "max_rel_err_vs_fp64": err, "clocks": res["clocks"]}
    hb.close()
    del res
    torch.cuda.empty_cache()
    return out


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------

def main():
    args = parse_args()
    if args.impl == "reference":
        return run_reference(args)
    if args.workload == "batch":
        return run_batch(args)
    import torch
    import spgemm_b200 as sg

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))

    wl = build_workload(args)
    stream = torch.cuda.current_stream()

    def to_dev(a, dt):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype=dt)

    handles, steps_fn, keep = [], None, []
    if args.workload == "galerkin":
        A, P = wl["A"], wl["P"]
        Ac = A.to_csc()
        tA = [to_dev(Ac.colptr, torch.int32), to_dev(Ac.rowidx, torch.int32), to_dev(Ac.val, torch.float32)]
        tP = [to_dev(P.rowptr, torch.int32), to_dev(P.col, torch.int32), to_dev(P.val, torch.float32)]
        keep += tA + tP
        A_cm = sg.device_cm(tA[0].data_ptr(), tA[1].data_ptr(), tA[2].data_ptr(), A.nnz, A.rows, A.cols, sg.COL_MAJOR)
        P_cm = sg.device_cm(tP[0].data_ptr(), tP[1].data_ptr(), tP[2].data_ptr(), P.nnz, P.rows, P.cols, sg.ROW_MAJOR)
        PT_cm = sg.device_cm(tP[0].data_ptr(), tP[1].data_ptr(), tP[2].data_ptr(), P.nnz, P.cols, P.rows, sg.COL_MAJOR)
        h1, h2 = sg.Handle(wl["precision"]), sg.Handle(wl["precision"])
        for h in (h1, h2):
            if tune_overrides(args):
                h.set_tuning(**tune_overrides(args))
        handles = [h1, h2]

        def step():
            AP = h1.multiply(A_cm, P_cm)
            h2.multiply(PT_cm, AP)
        ap_nnz = 0
        flops_per_step = None
    else:
        A, B = wl["products"][0]
        Ac = A.to_csc()
        tA = [to_dev(Ac.colptr, torch.int32), to_dev(Ac.rowidx, torch.int32), to_dev(Ac.val, torch.float32)]
        tB = [to_dev(B.rowptr, torch.int32), to_dev(B.col, torch.int32), to_dev(B.val, torch.float32)]
        keep += tA + tB
        A_cm = sg.device_cm(tA[0].data_ptr(), tA[1].data_ptr(), tA[2].data_ptr(), A.nnz, A.rows, A.cols, sg.COL_MAJOR)
        B_cm = sg.device_cm(tB[0].data_ptr(), tB[1].data_ptr(), tB[2].data_ptr(), B.nnz, B.rows, B.cols, sg.ROW_MAJOR)
        h1 = sg.Handle(wl["precision"])
        if tune_overrides(args):
            h1.set_tuning(**tune_overrides(args))
        handles = [h1]
        out = {}

        def step():
            nnz = h1.symbolic(A_cm, B_cm)
            if out.get("cap", -1) < nnz:  # first call only: same product every step
                out["rowptr"] = torch.empty(A.rows + 1, dtype=torch.int32, device=dev)
                out["col"] = torch.empty(max(nnz, 1), dtype=torch.int32, device=dev)
                out["val"] = torch.empty(max(nnz, 1), dtype=torch.float32, device=dev)
                out["cap"] = nnz
            h1.numeric(out["rowptr"].data_ptr(), out["col"].data_ptr(), out["val"].data_ptr())
    for h in handles:
        h.set_stream(stream.cuda_stream)
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device=dev)

    for _ in range(max(args.warmup, 0)):
        step()
    torch.cuda.synchronize()
    stats = [h.stats() for h in handles]
    products = sum(s["intermediate_products"] for s in stats)
    nnz_c = stats[-1]["nnz_c"]
    launches0 = sum(s["kernel_launches"] for s in stats)
    for h in handles:
        h.reset_kernel_times()
        h.set_profiling(True)

    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
    smi_id = vis.split(",")[local].strip() if vis else str(local)
    sampler = ClockSampler(smi_id) if rank == 0 else None
    if sampler:
        sampler.start()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps)]
    for k in range(args.steps):
        flush.zero_()
        ev[k][0].record(stream)
        step()
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    clocks = sampler.stop() if sampler else None
    step_ms = [a.elapsed_time(b) for a, b in ev]
    total_ms = float(sum(step_ms))
    launches = sum(h.stats()["kernel_launches"] for h in handles) - launches0
    ktimes = {}
    for h in handles:
        h.set_profiling(False)
        for name, (ms, cnt) in h.kernel_times().items():
            t = ktimes.get(name, (0.0, 0))
            ktimes[name] = (t[0] + ms, t[1] + cnt)
    if dist:
        t = torch.tensor([total_ms], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    flops = 2.0 * products * args.steps * world
    value = flops / (total_ms / 1e3) / 1e9
    peak, peak_kind = measured_peaks()

    # roofline of the dominant kernel + the whole pipeline
    roof, pipeline = None, None
    if args.workload != "galerkin" and rank == 0:
        A, B = wl["products"][0]
        p_i, a_len, b_touched, span = product_stats(A, B)
        crow = out["rowptr"].cpu().numpy()
        o_i = np.diff(crow.astype(np.int64))
        total_alg = algorithmic_bytes(np.ones(A.rows, bool), p_i, a_len, o_i, b_touched, products)
        step_s = total_ms / args.steps / 1e3
        pipeline = {"algorithmic_bytes": total_alg, "gbs": total_alg / step_s / 1e9 / world,
                    "frac": total_alg / step_s / 1e9 / world / peak,
                    "kernel_ms_per_step": {k: v[0] / args.steps for k, v in
                                           sorted(ktimes.items(), key=lambda kv: -kv[1][0])}}
        dom = max(ktimes.items(), key=lambda kv: kv[1][0]) if ktimes else None
        if dom:
            name, (ms, cnt) = dom
            sel, writes_c = kernel_rows(name, p_i, o_i, span, B.cols)
            if sel is not None:
                alg = algorithmic_bytes(sel, p_i, a_len, o_i, b_touched, products, with_c=writes_c)
                per_launch = alg * args.steps / cnt
                avg_s = ms / cnt / 1e3
                wl_key = f"rmat{args.scale}" if args.workload == "rmat" else args.workload
                roof = {"bound": "hbm", "kernel": name, "achieved": per_launch / avg_s / 1e9,
                        "peak": peak, "unit": "GB/s", "frac": per_launch / avg_s / 1e9 / peak,
                        "traffic": profiled_traffic(wl_key, name),
                        "algorithmic_bytes_per_launch": per_launch,
                        "avg_launch_ms": ms / cnt, "peak_kind": peak_kind}

    # e2e through the host-buffer C ABI (pinned host memory)
    e2e = None
    if not args.no_e2e and args.workload != "galerkin":
        A, B = wl["products"][0]
        Ac = A.to_csc()
        pin = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(dt).pin_memory()
        hA = [pin(Ac.colptr, torch.int32), pin(Ac.rowidx, torch.int32), pin(Ac.val, torch.float32)]
        hB = [pin(B.rowptr, torch.int32), pin(B.col, torch.int32), pin(B.val, torch.float32)]
        try:
            o_rp = torch.empty(A.rows + 1, dtype=torch.int32).pin_memory()
            o_col = torch.empty(nnz_c, dtype=torch.int32).pin_memory()
            o_val = torch.empty(nnz_c, dtype=torch.float32).pin_memory()
            pinned_out = True
        except RuntimeError:
            o_rp = torch.empty(A.rows + 1, dtype=torch.int32)
            o_col = torch.empty(nnz_c, dtype=torch.int32)
            o_val = torch.empty(nnz_c, dtype=torch.float32)
            pinned_out = False
        Ah = sg.Csc(A.rows, A.cols, hA[0].numpy(), hA[1].numpy(), hA[2].numpy())
        Bh = sg.Csr(B.rows, B.cols, hB[0].numpy(), hB[1].numpy(), hB[2].numpy())
        he = sg.Handle(wl["precision"])
        if tune_overrides(args):
            he.set_tuning(**tune_overrides(args))
        he.set_stream(stream.cuda_stream)
        h2d = sum(t.numel() * 4 for t in hA + hB)
        d2h = (A.rows + 1 + 2 * nnz_c) * 4
        he.multiply_host_to(Ah, Bh, o_rp.numpy(), o_col.numpy(), o_val.numpy())  # warm-up
        torch.cuda.synchronize()
        e_ms = []
        for _ in range(args.e2e_steps):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            flush.zero_()
            s.record(stream)
            he.multiply_host_to(Ah, Bh, o_rp.numpy(), o_col.numpy(), o_val.numpy())
            e.record(stream)
            torch.cuda.synchronize()
            e_ms.append(s.elapsed_time(e))
        he.close()
        e_total = float(sum(e_ms))
        if dist:
            t = torch.tensor([e_total], dtype=torch.float64, device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            e_total = float(t.item())
        e2e = {"value": 2.0 * products * len(e_ms) * world / (e_total / 1e3) / 1e9, "unit": "GFLOP/s",
               "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
               "ms_per_step": e_total / len(e_ms), "pinned_output": pinned_out}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        A, B = (wl["A"], wl["P"]) if args.workload == "galerkin" else wl["products"][0]
        cpu, _ = cpu_baseline(A, B, args.cpu_seconds)

    # the other configurations on the same line (one GPU; R-MAT's buffers freed first)
    configs = None
    if rank == 0 and world == 1 and args.workload == "rmat" and not args.no_configs:
        A, B = wl["products"][0]
        try:
            rmat_err = sampled_row_error(A, B, out["rowptr"], out["col"], out["val"])
        except Exception as e:
            rmat_err = {"unavailable": str(e)[:200]}
        for h in handles:
            h.close()
        handles = []
        out.clear()
        keep.clear()
        del flush
        torch.cuda.empty_cache()
        configs = {"rmat18": {"max_rel_err_vs_fp64": rmat_err, "precision": "plain"}}
        configs.update(run_suite(args, dev, stream, smi_id))

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": "GFLOP/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": total_ms / args.steps, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic (seeded generator; the reference's SuiteSparse/SNAP inputs are not available)",
                "config": dict(wl["config"], intermediate_products=products, nnz_c=nnz_c,
                               l2="flushed before every step (512 MiB write)",
                               parallelism=f"replicas x{world} (one independent product per GPU)"),
                "roofline": roof, "pipeline": pipeline, "cpu_baseline": cpu, "e2e": e2e,
                "clocks": clocks, "gpu_launches": launches,
                "step_ms": step_ms}
        if configs is not None:
            line["configs"] = configs
        print(json.dumps(line), flush=True)
    for h in handles:
        h.close()
    if dist:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
