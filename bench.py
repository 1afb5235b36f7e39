#!/usr/bin/env python
"""Benchmark: Chebyshev steps*nnz/s of one Kubo-Bastin sigma_xx(E) solve on a B200.

Workload (one "step" = one solve): honeycomb graphene, 128 x 128 cells (N = 32,768
sites), t = -2.7 eV, Anderson disorder W = 1.0 eV (seed 21), V_x = i (x_i - x_j) H_ij
(a = 1.42 A); 8 random-phase vectors (seed 22) as one block; 512 x 512 2D moments
(CorrelationExpansionMoments) and the FFT Bastin reconstruction at 1024 energies
(Kubo_solver_FFT), both from one pass of the recursion.  Synthetic, seeded inputs stand
in for operators read from files.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl linqt|reference]
                    [--precision fp64|mixed] [--workload kubo|supercell]

metric = (recursion steps per vector column: 2M) x (columns: R) x nnz(H, Hermitian-
expanded, diagonal included) / seconds.  value: device time of K solves with operators
and states resident in HBM (CUDA events on the launching stream, max over ranks);
e2e: the same through the host-pointer C ABI call with the states copied from pinned
host memory and mu / sigma(E) copied back inside the timed region.  Multi-GPU: one
independent solve per rank (different random vectors), no collective on the data path.

--workload supercell times the operator builder instead (LinQT's wannier2sparse): the
Hamiltonian of a synthetic 18-orbital Wannier model (hoppings to |R_i| <= 3, seed 7) on a
128 x 128 x 1 supercell, written as the upper-triangle CSR of LABEL.HAM.CSR.  metric =
stored entries / second; value: the device build into HBM-resident buffers; e2e: the model
files read and the CSR returned in pinned host arrays (linqt_supercell_csr) every step; the
reference arm runs the reference tool built from its sources on a bounded supercell.
"""
import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = dict(workload="kubo_bastin_graphene_128x128", lattice="honeycomb", Lx=128, Ly=128, t=-2.7, W=1.0, a=1.42,
                disorder_seed=21, phase_seed=22, R=8, M=512, nump=1024, formula="bastin", bounds_pad=1.05)
METRIC = "chebyshev_steps_nnz_per_s"
UNIT = "steps*nnz/s"


def build_inputs(rank=0):
    from linqt_b200 import lattices
    w = WORKLOAD
    N, H, V = lattices.honeycomb(w["Lx"], w["Ly"], t=w["t"], W=w["W"], seed=w["disorder_seed"], a=w["a"])
    lo, hi = lattices.gershgorin_bounds(N, *H)
    bw = w["bounds_pad"] * (hi - lo)
    bc = (hi + lo) / 2
    st = lattices.random_phase_states(N, w["R"], seed=w["phase_seed"] + 1000 * rank)
    return N, H, V, bw, bc, st


def max_over_ranks(x, dist, device):
    """The slowest rank's time (replicas run the same work; the job ends with the last)."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rates(units_per_rank, world, dev_ms, e2e_ms):
    """Whole-job throughput: all ranks' units over the max-over-ranks times."""
    return world * units_per_rank / (dev_ms * 1e-3), world * units_per_rank / (e2e_ms * 1e-3)


def nnz_full(N, H):
    rp, col, _ = H
    rows = np.repeat(np.arange(N), np.diff(rp))
    off = int((col != rows).sum())
    return N + 2 * off  # diagonal always present after rescaling


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                                       "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.f,
                                      stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.p:
            self.p.terminate()
            self.p.wait()

    def summary(self):
        self.f.seek(0)
        rows = [r.split(",") for r in self.f.read().strip().splitlines() if r.strip()]
        os.unlink(self.f.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if len(r) > 5 + i and "Active" in r[5 + i]
                          and "Not" not in r[5 + i]})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "samples": len(rows), "reasons": reasons}


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return d.get("hbm_gbs", 6650.0), d.get("bf16_tflops", 1590.0), "measured"
    return 6650.0, 1590.0, "fallback"


def fp64_peak_tflops(torch, device):
    """FP64 dense peak measured here with torch.matmul (cuBLAS DGEMM), best of 5."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device=device)
    b = torch.randn(n, n, dtype=torch.float64, device=device)
    for _ in range(2):
        a @ b
    best = 0.0
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        a @ b
        e1.record()
        e1.synchronize()
        best = max(best, 2 * n ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e12)
    del a, b
    return best


def run_reference(args):
    """The reference's own CPU solvers (oracle/_ref/ref_harness, LinQT's src/*.cpp built here)
    on a bounded sample: one of the 8 random vectors per step, the full M = 512, nump = 1024."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as orc
    from linqt_b200 import formats
    if not orc.ref_available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref is not built (needs the reference checkout)"}))
        return
    N, H, V, bw, bc, st = build_inputs(0)
    w = WORKLOAD
    d = tempfile.mkdtemp(prefix="linqt_bench_ref_")
    os.makedirs(os.path.join(d, "operators"))
    formats.write_csr(os.path.join(d, "operators", "gr.HAM.CSR"), N, *H)
    formats.write_csr(os.path.join(d, "operators", "gr.VX.CSR"), N, *V)
    lo, hi = bc - bw / 2, bc + bw / 2
    open(os.path.join(d, "BOUNDS"), "w").write("%.17g %.17g\n" % (lo, hi))
    threads = os.cpu_count() or 1
    nnz = nnz_full(N, H)
    total_s, total_units = 0.0, 0.0
    for it in range(args.warmup + args.steps):
        col = it % w["R"]
        sp = os.path.join(d, "st%d.txt" % col)
        if not os.path.exists(sp):
            formats.write_vector_states(sp, st[col:col + 1])
        a = orc.run_ref_harness(["nonEq", "gr", "VX", "VX", w["M"], os.path.basename(sp)], d, threads=threads)
        b = orc.run_ref_harness(["kuboFFT", "gr", "VX", "VX", w["M"], w["nump"], 1, os.path.basename(sp)], d,
                                threads=threads)
        if it >= args.warmup:
            total_s += a["seconds"] + b["seconds"]
            total_units += 2 * w["M"] * 1 * nnz
    value = total_units / total_s
    cfg = dict(WORKLOAD)
    cfg.update(parallelism="cpu", l2="n/a (CPU)")
    sample = "1 of the 8 random vectors per step (M=512, nump=1024): CorrelationExpansionMoments + Kubo_solver_FFT"
    print(json.dumps({"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
                      "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total_s / args.steps,
                      "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
                      "data": "synthetic (seeded)", "config": cfg,
                      "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "reference",
                                       "sample": sample},
                      "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}))


def cpu_baseline_sample():
    """Reference CPU solvers on one random vector of the same workload (rank 0, N=1 only)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as orc
    from linqt_b200 import formats
    if not orc.ref_available():
        return None
    N, H, V, bw, bc, st = build_inputs(0)
    w = WORKLOAD
    d = tempfile.mkdtemp(prefix="linqt_cpu_")
    os.makedirs(os.path.join(d, "operators"))
    formats.write_csr(os.path.join(d, "operators", "gr.HAM.CSR"), N, *H)
    formats.write_csr(os.path.join(d, "operators", "gr.VX.CSR"), N, *V)
    open(os.path.join(d, "BOUNDS"), "w").write("%.17g %.17g\n" % (bc - bw / 2, bc + bw / 2))
    formats.write_vector_states(os.path.join(d, "st.txt"), st[:1])
    threads = os.cpu_count() or 1
    a = orc.run_ref_harness(["nonEq", "gr", "VX", "VX", w["M"], "st.txt"], d, threads=threads)
    b = orc.run_ref_harness(["kuboFFT", "gr", "VX", "VX", w["M"], w["nump"], 1, "st.txt"], d, threads=threads)
    secs = a["seconds"] + b["seconds"]
    res = {"value": 2 * w["M"] * nnz_full(N, H) / secs, "unit": UNIT, "cores": threads, "kind": "reference",
           "sample": "1 of 8 random vectors, M=512, nump=1024 (CorrelationExpansionMoments %.2fs + "
                     "Kubo_solver_FFT %.2fs)" % (a["seconds"], b["seconds"])}
    # the reference's results for that vector: the parity check of the timed configuration
    _, _, _, mu_ref = formats.read_chebmom2d(os.path.join(d, a["out"]))
    sig_ref = np.loadtxt(os.path.join(d, b["out"]))
    return res, (mu_ref, sig_ref)


SC_WORKLOAD = dict(workload="supercell_wannier18_r3_128x128", model="synthetic Wannier90 model", orbitals=18, reach=3,
                   seed=7, cell_dim=[128, 128, 1], op="HAM", reference_cell_dim=[16, 16, 1])
SC_METRIC = "supercell_csr_entries_per_s"
SC_UNIT = "entries/s"


def supercell_inputs():
    from linqt_b200 import lattices
    d = tempfile.mkdtemp(prefix="linqt_w2s_")
    label = os.path.join(d, "syn")
    lattices.wannier_model(label, SC_WORKLOAD["orbitals"], SC_WORKLOAD["reach"], SC_WORKLOAD["seed"])
    return d, label


def supercell_reference_sample():
    """The reference tool (oracle/_ref/wannier2sparse, LinQT's utilities/wannier2sparse built
    here) on the bounded supercell: (entries/s, seconds, entries)."""
    tool = os.path.join(ROOT, "oracle", "_ref", "wannier2sparse")
    if not os.path.exists(tool):
        return None
    d, label = supercell_inputs()
    cd = [str(x) for x in SC_WORKLOAD["reference_cell_dim"]]
    t0 = time.perf_counter()
    subprocess.run([tool, "syn"] + cd, cwd=d, check=True, stdout=subprocess.DEVNULL)
    secs = time.perf_counter() - t0
    with open(os.path.join(d, "syn.HAM.CSR")) as f:
        nnz = int(f.readline().split()[1])
    return nnz / secs, secs, nnz


def run_supercell_reference(args):
    first = supercell_reference_sample()
    if first is None:
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/wannier2sparse is not built "
                                                              "(needs the reference checkout)"}))
        return
    secs = 0.0
    ents = 0
    for it in range(args.warmup + args.steps - 1):
        r = supercell_reference_sample()
        if it >= args.warmup - 1:
            secs += r[1]
            ents += r[2]
    value = ents / secs
    sample = "supercell %s of the same model (one thread: the tool is serial), text file included" % (
        "x".join(str(x) for x in SC_WORKLOAD["reference_cell_dim"]))
    print(json.dumps({"impl": "reference", "metric": SC_METRIC, "value": value, "unit": SC_UNIT, "n_gpus": args.gpus,
                      "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * secs / args.steps,
                      "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
                      "data": "synthetic (seeded model files)", "config": dict(SC_WORKLOAD, parallelism="cpu"),
                      "cpu_baseline": {"value": value, "unit": SC_UNIT, "cores": 1, "kind": "reference",
                                       "sample": sample},
                      "e2e": {"value": value, "unit": SC_UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}))


def run_supercell(args, rank, world, local):
    import torch
    import linqt_b200 as lq
    from linqt_b200._lib import check
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=torch.device("cuda", local))

    def barrier():
        if dist is not None:
            dist.barrier()

    w = SC_WORKLOAD
    d, label = supercell_inputs()
    stream = torch.cuda.current_stream()
    sess = lq.Session(local)
    sess.set_stream(stream)
    m = lq.TBModel.load(label)
    dims, op = w["cell_dim"], w["op"]
    n, nnz = m.csr_size(op, dims, session=sess)
    rp = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    cl = torch.empty(nnz, dtype=torch.int32, device="cuda")
    vl = torch.empty(2 * nnz, dtype=torch.float64, device="cuda")

    def build():
        m.supercell_csr_dev(op, dims, rp, cl, vl, nnz, session=sess)

    for _ in range(args.warmup):
        build()
    torch.cuda.synchronize()
    sess.enable_timing(True)
    sess.phase_times(reset=True)
    with ClockSampler(local) as clocks:
        barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            build()
        e1.record(stream)
        torch.cuda.synchronize()
        barrier()
    dev_ms = e0.elapsed_time(e1) / args.steps
    phase_ms, phase_launches = sess.phase_times(reset=True)
    sess.enable_timing(False)
    clk = clocks.summary()

    # end to end: read the model files and return the CSR in (pinned) host arrays, every step
    out_rp = torch.empty(n + 1, dtype=torch.int32).pin_memory()
    out_cl = torch.empty(nnz, dtype=torch.int32).pin_memory()
    out_vl = torch.empty(2 * nnz, dtype=torch.float64).pin_memory()

    def build_host():
        mm = lq.TBModel.load(label)
        nn, kk = ctypes.c_int(), ctypes.c_long()
        dd = np.ascontiguousarray(dims, dtype=np.int32)
        check(lq.load().linqt_supercell_csr(sess.h, mm.h, op.encode(),
                                               dd.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), ctypes.byref(nn),
                                               ctypes.byref(kk), ctypes.cast(out_rp.data_ptr(), ctypes.POINTER(ctypes.c_int)),
                                               ctypes.cast(out_cl.data_ptr(), ctypes.POINTER(ctypes.c_int)),
                                               ctypes.cast(out_vl.data_ptr(), ctypes.POINTER(ctypes.c_double)), nnz))
        mm.close()

    import ctypes
    build_host()
    barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        build_host()
    torch.cuda.synchronize()
    barrier()
    e2e_ms = 1e3 * (time.perf_counter() - t0) / args.steps
    assert torch.equal(out_rp, rp.cpu()) and torch.equal(out_cl, cl.cpu()) and torch.equal(out_vl, vl.cpu())

    dev_ms = max_over_ranks(dev_ms, dist, "cuda")
    e2e_ms = max_over_ranks(e2e_ms, dist, "cuda")
    value, e2e = whole_job_rates(nnz, world, dev_ms, e2e_ms)
    hbm_peak, _, peak_src = measured_peaks()
    out_bytes = 20 * nnz + 4 * (n + 1)
    ach = out_bytes / (dev_ms * 1e-3) / 1e9
    roof = {"kernel": "k_row_totals + k_scan_totals + k_rowptr + k_fill (whole build)", "bound": "hbm",
            "achieved": ach, "peak": hbm_peak, "unit": "GB/s", "frac": ach / hbm_peak, "peak_source": peak_src,
            "algorithmic_bytes": "20 B per stored entry (int32 column + complex128 value) + 4 B per row pointer",
            "traffic": None}
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            r = supercell_reference_sample()
            if r:
                cpu = {"value": r[0], "unit": SC_UNIT, "cores": 1, "kind": "reference",
                       "sample": "reference tool on the %s supercell of the same model (%.1f s, %d entries, "
                                 "text file included)" % ("x".join(str(x) for x in w["reference_cell_dim"]), r[1],
                                                          r[2])}
        except Exception as ex:
            cpu = {"error": str(ex)[:200]}
    if rank == 0:
        cfg = dict(w, parallelism="replicas%d" % world if world > 1 else "single", N=n, nnz_upper=nnz,
                   l2="output larger than L2: %.1f GB written per build" % (out_bytes / 1e9))
        print(json.dumps({"metric": SC_METRIC, "value": value, "unit": SC_UNIT, "n_gpus": world, "steps": args.steps,
                          "warmup": args.warmup, "ms_per_step": dev_ms, "higher_is_better": True, "scaling": "weak",
                          "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded model files)",
                          "config": cfg,
                          "e2e": {"value": e2e, "unit": SC_UNIT, "ms_per_step": e2e_ms,
                                  "h2d_bytes_per_step": int(os.path.getsize(label + "_hr.dat")),
                                  "d2h_bytes_per_step": int(out_bytes)},
                          "gpu_launches": int(sum(phase_launches)), "roofline": roof,
                          "build_phases_ms": round(phase_ms[3] / args.steps, 4), "clocks": clk,
                          "cpu_baseline": cpu}))
    if dist is not None:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="linqt", choices=["linqt", "reference"])
    ap.add_argument("--precision", default="fp64", choices=["fp64", "mixed", "fp32"])
    ap.add_argument("--format", default="auto", choices=["csr", "sell", "auto"],
                    help="sparse layout of the recursion (auto: layout and thread shape tuned in the warm-up)")
    ap.add_argument("--no-compare", action="store_true", help="skip the mixed-vs-FP64 accuracy run")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--workload", default="kubo", choices=["kubo", "supercell"])
    ap.add_argument("--sc-cells", type=int, default=None, help="supercell: L x L x 1 cells (profiling captures)")
    # size overrides, for profiling captures on a smaller case of the same kernels
    ap.add_argument("--lx", type=int, default=None)
    ap.add_argument("--ly", type=int, default=None)
    ap.add_argument("--moments", type=int, default=None)
    ap.add_argument("--vectors", type=int, default=None)
    args = ap.parse_args()
    for k, v in (("Lx", args.lx), ("Ly", args.ly), ("M", args.moments), ("R", args.vectors)):
        if v:
            WORKLOAD[k] = v
            WORKLOAD["workload"] = "kubo_bastin_graphene_%dx%d_M%d_R%d" % (WORKLOAD["Lx"], WORKLOAD["Ly"],
                                                                         WORKLOAD["M"], WORKLOAD["R"])
    args.warmup = max(args.warmup, 3)

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if args.workload == "supercell":
        if args.sc_cells:
            SC_WORKLOAD["cell_dim"] = [args.sc_cells, args.sc_cells, 1]
            SC_WORKLOAD["workload"] = "supercell_wannier18_r3_%dx%d" % (args.sc_cells, args.sc_cells)
        if args.impl == "reference":
            if rank == 0:
                run_supercell_reference(args)
            return
        run_supercell(args, rank, world, local)
        return

    if args.impl == "reference":
        if rank == 0:
            run_reference(args)
        return

    import torch
    import linqt_b200 as lq

    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=torch.device("cuda", local))

    w = WORKLOAD
    N, H, V, bw, bc, st = build_inputs(rank)
    nnz = nnz_full(N, H)
    M, R, nump = w["M"], w["R"], w["nump"]
    stream = torch.cuda.current_stream()
    sess = lq.Session(local)
    sess.set_stream(stream)
    Hg = lq.Operator.from_csr(N, *H, session=sess)
    Hg.rescale_to_chebyshev(bw, bc)
    Vg = lq.Operator.from_csr(N, *V, session=sess)
    assert Hg.nnz == nnz
    prec = {"fp64": lq.PREC_FP64, "mixed": lq.PREC_MIXED, "fp32": lq.PREC_FP32}[args.precision]
    fmt = {"csr": 0, "sell": 1, "auto": 2}[args.format]
    opts = lq.make_opts(precision=prec, fmt=fmt)

    st_dev = torch.from_numpy(st.view(np.float64).copy()).cuda()
    mu_dev = torch.zeros(2 * M * M, dtype=torch.float64, device="cuda")
    out_dev = torch.zeros(3 * nump, dtype=torch.float64, device="cuda")

    def solve_dev():
        lq.kubo_bastin_dev(Hg, Vg, Vg, st_dev, R, M, nump, bw, bc, mu_dev, out_dev, opts=opts, session=sess)

    for _ in range(args.warmup):
        solve_dev()
    torch.cuda.synchronize()
    sess.enable_timing(True)
    sess.phase_times(reset=True)

    def barrier():
        if dist is not None:
            dist.barrier()

    with ClockSampler(local) as clocks:
        barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            solve_dev()
        e1.record(stream)
        torch.cuda.synchronize()
        barrier()
    dev_ms = e0.elapsed_time(e1) / args.steps
    phase_ms, phase_launches = sess.phase_times(reset=True)
    sess.enable_timing(False)
    clk = clocks.summary()

    # ---- end to end through the host-pointer C ABI call (pinned host buffers)
    st_pin = torch.from_numpy(st.view(np.float64).copy()).pin_memory()
    mu_pin = torch.zeros(2 * M * M, dtype=torch.float64).pin_memory()
    E_pin = torch.zeros(nump, dtype=torch.float64).pin_memory()
    s_pin = torch.zeros(nump, dtype=torch.float64).pin_memory()

    def solve_host():
        lq.kubo_bastin_host_ptr(Hg, Vg, Vg, st_pin.data_ptr(), R, M, nump, bw, bc, mu_pin.data_ptr(), E_pin.data_ptr(),
                                s_pin.data_ptr(), opts=opts, session=sess)

    for _ in range(max(3, args.warmup)):  # as many untimed calls as the device-timed loop
        solve_host()
    barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        solve_host()
    torch.cuda.synchronize()
    barrier()
    e2e_ms = 1e3 * (time.perf_counter() - t0) / args.steps

    dev_ms = max_over_ranks(dev_ms, dist, "cuda")
    e2e_ms = max_over_ranks(e2e_ms, dist, "cuda")
    units = 2 * M * R * nnz  # recursion steps x nnz per solve and rank
    value, e2e = whole_job_rates(units, world, dev_ms, e2e_ms)

    # ---- roofline of the dominant phase
    hbm_peak, bf16_peak, peak_src = measured_peaks()
    K = N * R
    esz = 16 if prec == lq.PREC_FP64 else 8
    rec_bytes_per_step = nnz * (16 + 4) + 4 * (N + 1) + 3 * 16 * N * R
    phases = {
        "recursion": {"ms": phase_ms[0] / args.steps, "launches": phase_launches[0] // args.steps,
                      "bytes": 2 * M * rec_bytes_per_step},
        "contraction": {"ms": phase_ms[1] / args.steps, "launches": phase_launches[1] // args.steps,
                        "flops": 8.0 * M * M * K},
        "fft": {"ms": phase_ms[2] / args.steps, "launches": phase_launches[2] // args.steps,
                "flops": 8.0 * K * 5 * nump * np.log2(nump)},
        "other": {"ms": phase_ms[3] / args.steps, "launches": phase_launches[3] // args.steps},
    }
    fp64_peak = fp64_peak_tflops(torch, "cuda")
    dom = max(("recursion", "contraction", "fft"), key=lambda k: phases[k]["ms"])
    if dom == "recursion":
        ach = phases[dom]["bytes"] / (phases[dom]["ms"] * 1e-3) / 1e9
        roof = {"kernel": "cheb_step (recursion)", "bound": "hbm", "achieved": ach, "peak": hbm_peak, "unit": "GB/s",
                "frac": ach / hbm_peak, "peak_source": peak_src}
    else:
        ach = phases[dom]["flops"] / (phases[dom]["ms"] * 1e-3) / 1e12
        roof = {"kernel": {"contraction": "mu_nm contraction", "fft": "kubo_fft (per-site DFTs)"}[dom],
                "bound": "tensor", "pipe": "fp64", "achieved": ach, "peak": fp64_peak, "unit": "TFLOP/s",
                "frac": ach / fp64_peak, "peak_source": "FP64 DGEMM (torch.matmul 8192^3) measured in this run"}
        if dom == "contraction" and prec == lq.PREC_FP64:
            # the complex FP64 product runs as 34 exact INT8 products (17 moduli, two real products each);
            # the phase also holds the residues and the Chinese remainders
            ops = 34 * 2.0 * M * M * K / (phases[dom]["ms"] * 1e-3) / 1e12
            roof.update(kernel="k_residues, k_rns_gemm, k_rns_crt (mu_nm contraction)", pipe="int8", achieved=ops,
                        peak=2 * bf16_peak, unit="TOP/s", frac=ops / (2 * bf16_peak),
                        peak_source="twice the measured bf16 GEMM rate", algorithmic_fp64_tflops=ach)
    # DRAM bytes per launch of the per-site transforms: ncu capture of the 64x64-cell case
    # (M = 256, K = 65,536; dram__bytes_read.sum + dram__bytes_write.sum), scaled by M*K,
    # which their operand reads are proportional to
    traffic_per_mk = {"fft": (545405952 + 114432) / (256 * 65536)}
    roof["traffic"] = (traffic_per_mk[dom] * M * K) if dom in traffic_per_mk else None
    roof["traffic_unit"] = "bytes per launch (scaled from the 64x64-cell ncu capture)"
    rec_ach = phases["recursion"]["bytes"] / (phases["recursion"]["ms"] * 1e-3) / 1e9
    for k in phases:
        phases[k]["ms"] = round(phases[k]["ms"], 4)

    # ---- the other precision on the same inputs: throughput and accuracy against FP64
    other = None
    if not args.no_compare:
        other_prec = lq.PREC_MIXED if prec == lq.PREC_FP64 else lq.PREC_FP64
        oopts = lq.make_opts(precision=other_prec, fmt=fmt)
        mu_o = torch.zeros_like(mu_dev)
        out_o = torch.zeros_like(out_dev)

        def solve_other():
            lq.kubo_bastin_dev(Hg, Vg, Vg, st_dev, R, M, nump, bw, bc, mu_o, out_o, opts=oopts, session=sess)

        for _ in range(args.warmup):
            solve_other()
        torch.cuda.synchronize()
        sess.enable_timing(True)
        sess.phase_times(reset=True)
        barrier()
        torch.cuda.synchronize()
        f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        for _ in range(args.steps):
            solve_other()
        f1.record(stream)
        torch.cuda.synchronize()
        barrier()
        o_ms = max_over_ranks(f0.elapsed_time(f1) / args.steps, dist, "cuda")
        o_phase, o_launch = sess.phase_times(reset=True)
        sess.enable_timing(False)
        solve_dev()
        torch.cuda.synchronize()
        mu64 = (mu_dev if prec == lq.PREC_FP64 else mu_o).cpu().numpy().view(np.complex128)
        mulo = (mu_o if prec == lq.PREC_FP64 else mu_dev).cpu().numpy().view(np.complex128)
        s64 = (out_dev if prec == lq.PREC_FP64 else out_o).cpu().numpy()[nump:2 * nump]
        slo = (out_o if prec == lq.PREC_FP64 else out_dev).cpu().numpy()[nump:2 * nump]
        lo_i, hi_i = int(0.05 * nump), int(0.95 * nump)  # interior 90 % of the energy window
        err_sigma = float(np.abs(slo - s64)[lo_i:hi_i].max() / np.abs(s64[lo_i:hi_i]).max())
        err_mu = float(np.abs(mulo - mu64).max() / np.abs(mu64).max())
        name = "mixed" if other_prec == lq.PREC_MIXED else "fp64"
        other = {"precision": name, "value": world * units / (o_ms * 1e-3), "ms_per_step": o_ms,
                 "phases_ms": {k: round(v / args.steps, 4) for k, v in zip(("recursion", "contraction", "fft", "other"),
                                                                           o_phase)},
                 "err_mu_vs_fp64": err_mu, "err_sigma_vs_fp64_interior90": err_sigma,
                 "dtype": "f32 recursion vectors (f64 operators and accumulation) + tcgen05 INT8 contraction of "
                          "4-digit splits with exact INT32 accumulation, FP64 across chunks + FP64 FFT"
                          if name == "mixed" else "f64"}
        # tensor-pipe view of the tcgen05 contraction: 10 digit products x real GEMM (2M x M x 2K MACs)
        if name == "mixed" and o_phase[1] > 0:
            tc_ops = 10 * 2.0 * (2 * M) * M * (2 * K)
            other["contraction_int8_tops"] = tc_ops / (o_phase[1] / args.steps * 1e-3) / 1e12

    cpu, parity = None, None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            sample = cpu_baseline_sample()
        except Exception as ex:  # report, do not fail the GPU measurement
            sample, cpu = None, {"error": str(ex)[:200]}
        if sample is not None:
            cpu, (mu_ref, sig_ref) = sample
            # the same solve on the GPU for that vector alone, in the precision timed above
            mu1, (E1, s1, _) = lq.kubo_bastin(Hg, Vg, Vg, st[:1], M, nump, bw, bc, opts=opts, session=sess)
            lo_i, hi_i = int(0.05 * nump), int(0.95 * nump)
            parity = {"against": "the reference's CorrelationExpansionMoments and Kubo_solver_FFT (oracle/_ref) "
                                 "on random vector 0 of the timed configuration",
                      "mu_max_rel_err": float(np.abs(mu1 - mu_ref).max() / np.abs(mu_ref).max()),
                      "mu_printed_digits": 15,
                      "sigma_max_rel_err_interior90": float(np.abs(s1 - sig_ref[:, 1])[lo_i:hi_i].max()
                                                            / np.abs(sig_ref[lo_i:hi_i, 1]).max()),
                      "sigma_printed_digits": 6}

    if rank == 0:
        cfg = dict(WORKLOAD)
        cfg.update(parallelism="replicas%d" % world if world > 1 else "single",
                   l2="inputs larger than L2: 4.3 GB of Chebyshev blocks written and read per solve",
                   nnz_full=nnz, N=N)
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": dev_ms, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "f64" if prec == lq.PREC_FP64 else "f32+int8x4",
                "data": "synthetic (seeded lattice, random-phase states)", "config": cfg,
                "e2e": {"value": e2e, "unit": UNIT, "ms_per_step": e2e_ms,
                        "h2d_bytes_per_step": int(st.nbytes), "d2h_bytes_per_step": int(16 * M * M + 16 * nump)},
                "gpu_launches": int(sum(phase_launches) // args.steps * args.steps),
                "roofline": roof,
                "roofline_recursion": {"bound": "hbm", "achieved": rec_ach, "peak": hbm_peak, "unit": "GB/s",
                                       "frac": rec_ach / hbm_peak, "peak_source": peak_src},
                "phases": phases, "fp64_peak_tflops": fp64_peak, "clocks": clk, "cpu_baseline": cpu,
                "parity": parity,
                "other_precision": other}
        print(json.dumps(line))
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
