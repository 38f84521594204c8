#!/usr/bin/env python
"""Benchmark of the B200 Smith-Waterman hot path (banded seed extension).

Workload (one step): config 1 -- the left (reversed prefix) and right
extensions of 5M synthetic 150 bp reads per GPU off a seeded 100 Mbp
reference with 20% of reads from tandem-repeat blocks (~10M extension
tasks), every task bit-exact with BandedSWScalar.align.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

value    extensions/s with inputs resident in HBM (swb_ext_batch_device),
         timed with CUDA events on the launching stream, max over ranks.
e2e      the same metric through the C ABI's host entry point
         (swb_ext_batch) from pinned host buffers: H2D of reads + tasks,
         the kernels, D2H of results, every step.
roofline the int ops (13 per DP cell) of the cells that a timed step computes
         / its time, against the packed 16-bit DPX add/max rate of the same GPU
         in lane operations (swb_int16x2_alu_peak; int32_frac: against
         swb_int_alu_peak).  Rows that cannot change a result are left out of
         the timed steps; every_row_pass is the profiled pass that computes
         them, whose cells (gcups) are the reference's.
For N > 1 the driver launches one process per GPU (torchrun); each rank
extends its own shard (weak scaling, no data-path collective).
"""
from __future__ import annotations

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

OPS_PER_CELL_EXT = 13   # add q, select M!=0, 2 max for H, 2x{sub,max0,sub,max} for E/F, 1 row-max


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--n-reads", type=int, default=5_000_000)
    ap.add_argument("--ref-len", type=int, default=100_000_000)
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="target CPU-baseline sample time")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-suite", action="store_true", help="skip the configs 0/2/3/4 and NW measurements")
    ap.add_argument("--serve-seconds", type=float, default=5.0)
    ap.add_argument("--c2-tasks", type=int, default=20_000_000)
    ap.add_argument("--c3-pairs", type=int, default=2_000_000)
    ap.add_argument("--nw-reads", type=int, default=1_000_000)
    ap.add_argument("--c4-ref-len", type=int, default=1_000_000_000)
    ap.add_argument("--c4-pool", type=int, default=3_000_000)
    ap.add_argument("--sat-requests", type=int, default=120)
    ap.add_argument("--c4-wave", type=int, default=1 << 17, help="served mode: tasks per wave")
    ap.add_argument("--c4-latency-cells", type=int, default=0,
                    help="served mode: tasks above this many DP cells run one warp per extension")
    ap.add_argument("--c5-chains", type=int, default=1_000_000)
    ap.add_argument("--no-tune", action="store_true", help="keep the default length classes (no autotuning)")
    ap.add_argument("--tune-sample", type=int, default=0,
                    help="tasks the length-class autotuner times (0: the whole workload)")
    ap.add_argument("--c3-jobs", type=int, default=1_000_000)
    ap.add_argument("--seed-reads", type=int, default=1_000_000, help="seeding: config-1 reads per SMEM batch")
    ap.add_argument("--suite-only", default="",
                    help="comma list of secondary configs to run alone (config0, config2, config3, config3_rescue_driver, "
                         "config1_nw_cigar, config5_extend_chains, seeding, config4); prints their JSON and skips "
                         "the headline")
    return ap.parse_args()


# ----------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except FileNotFoundError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if not self.proc:
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
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


# --------------------------------------------------------------- helpers
from swiftbwa_b200.sharding import dist_env, max_over_ranks, whole_job_rate  # noqa: E402


def traffic_per_launch(kernel: str):
    """Per-launch DRAM bytes (read + write) of `kernel` from the committed ncu summary."""
    p = os.path.join(ROOT, "profiles", "ncu_traffic.json")
    if not os.path.exists(p):
        return None
    try:
        d = json.load(open(p))
        return d.get(kernel, {}).get("dram_bytes_per_launch_full_workload")
    except Exception:
        return None


def cpu_baseline(wl, sc, seconds: float, gpu_out=None):
    """The oracle (C++ restatement of the reference's CPU code) on a bounded
    sample of the same tasks, all host threads."""
    from oracle import oracle
    threads = os.cpu_count() or 1
    n = len(wl.tasks)
    probe = min(n, 20_000)
    t0 = time.perf_counter()
    oracle.ext_batch(sc, wl.bases, wl.tasks[:probe], pac=wl.ref.pac, ref_bases=wl.ref.n, n_threads=threads)
    rate = probe / max(time.perf_counter() - t0, 1e-6)
    s = int(min(n, max(probe, rate * seconds)))
    t0 = time.perf_counter()
    res, cells = oracle.ext_batch(sc, wl.bases, wl.tasks[:s], pac=wl.ref.pac, ref_bases=wl.ref.n,
                                  n_threads=threads)
    dt = time.perf_counter() - t0
    out = {"value": s / dt, "unit": "ext/s", "cores": threads, "kind": "port",
           "sample": f"first {s} of {n} config-1 extension tasks ({cells} DP cells, {dt:.1f} s)",
           "gcups": cells / dt / 1e9}
    if gpu_out is not None:
        same = int(np.sum(np.all(np.stack([gpu_out[f][:s] == res[f] for f in res.dtype.names]), axis=0)))
        out["bitexact_sample"] = f"{same}/{s}"
    return out


# -------------------------------------------------------- secondary suite
def _cuda_time(torch, stream, fn, reps):
    """Average device ms of fn() over reps calls (events on `stream`)."""
    fn()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        fn()
    e1.record(stream)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def _warm_server(S, srv, pb, pt, po, reqs):
    """Runs the stream's largest requests once so that a fresh server's lanes
    have grown their buffers before anything is timed."""
    big = sorted(reqs, key=lambda r: r.hi - r.lo)[-4:]
    S.run_pool_stream(srv, pb, pt, po, [S.Request(r.lo, r.hi, 0.0) for r in big], open_loop=False)


def _pct(xs, q):
    return float(np.percentile(np.asarray(xs), q)) if len(xs) else None


def secondary_suite(eng, sc, args, dev, torch, cpu_on=True, only=None):
    """Configs 0, 2, 3, 4, 5 and the config-1 NW+CIGAR stage, each bounded to a
    few seconds of GPU time; CPU-oracle samples beside them."""
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.abi import (EXT_RESULT_DTYPE, CIGAR_RESULT_DTYPE, CIGAR_TASK_DTYPE, LOCAL_RESULT_DTYPE,
                                   REGION_DTYPE, SMEM_DTYPE)
    from oracle import oracle
    threads = os.cpu_count() or 1
    out = {}

    def want(name):
        return only is None or name in only

    stream = torch.cuda.Stream(dev)

    # ---- config 0: 10k right extensions (host entry point; launch-latency bound)
    if want("config0"):
        wl0 = W.config0()
        eng.upload_reference(wl0.ref.pac, wl0.ref.n)
        eng.ext_batch(sc, wl0.bases, wl0.tasks)
        t0 = time.perf_counter()
        for _ in range(5):
            r0 = eng.ext_batch(sc, wl0.bases, wl0.tasks)
        e2e0 = (time.perf_counter() - t0) / 5
        ms0, cells0 = eng.last_batch_stats()
        exp0, _ = oracle.ext_batch(sc, wl0.bases, wl0.tasks, pac=wl0.ref.pac, ref_bases=wl0.ref.n, n_threads=threads)
        out["config0"] = {"tasks": len(wl0.tasks), "e2e_ext_per_s": len(wl0.tasks) / e2e0, "kernel_ms": ms0,
                          "gcups_kernel": cells0 / ms0 / 1e6, "bitexact": bool(np.array_equal(r0, exp0))}

    # ---- config 2: 20M uneven extensions, binned (ours) vs the plain single-launch kernel
    if want("config2"):
        wl2 = W.config2(n=args.c2_tasks)
        eng.upload_reference(wl2.ref.pac, wl2.ref.n)
        tune2 = None if args.no_tune else eng.tune_ext_bins(sc, wl2.bases, wl2.tasks[: args.tune_sample or None])
        db = torch.from_numpy(wl2.bases).to(dev)
        dt = torch.from_numpy(wl2.tasks.view(np.uint8)).to(dev)
        n2 = len(wl2.tasks)
        do = torch.empty(n2 * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8, device=dev)
        do2 = torch.empty_like(do)
        torch.cuda.synchronize()
        def binned():
            eng.ext_batch_device(sc, db.data_ptr(), dt.data_ptr(), n2, do.data_ptr(), stream.cuda_stream)
        ms_b = _cuda_time(torch, stream, binned, 2)
        eng.profile(True)       # the reference's cell count, from a pass outside the timing
        eng.profile_reset()
        binned()
        prof2 = eng.profile_read()
        eng.profile(False)
        cells2 = sum(v[2] for k, v in prof2.items() if k.startswith("ext_"))
        def plain():
            eng.ext_batch_plain_device(sc, db.data_ptr(), dt.data_ptr(), n2, do2.data_ptr(), stream.cuda_stream)
        ms_p = _cuda_time(torch, stream, plain, 2)
        same2 = bool(torch.equal(do, do2))
        c2 = {"tasks": n2, "binned_ms": ms_b, "binned_ext_per_s": n2 / ms_b * 1e3, "gcups": cells2 / ms_b / 1e6,
              "plain_kernel_ms": ms_p, "plain_kernel_ext_per_s": n2 / ms_p * 1e3, "speedup_vs_plain": ms_p / ms_b,
              "plain_kernel": "swb_ext_batch_plain_device: the same two-row kernel, one launch over the batch in "
                              "input order (one task per thread, no sort, bins or claiming), rows sized to the "
                              "batch's longest query",
              "binned_equals_plain": same2, "ext_bins": eng.ext_bins(), "ext_bins_tuning": tune2}
        if cpu_on:
            s2 = 60_000
            t0 = time.perf_counter()
            e2, _ = oracle.ext_batch(sc, wl2.bases, wl2.tasks[:s2], pac=wl2.ref.pac, ref_bases=wl2.ref.n, n_threads=threads)
            c2["cpu_baseline"] = {"value": s2 / (time.perf_counter() - t0), "unit": "ext/s", "cores": threads, "kind": "port",
                                  "sample": f"first {s2} tasks"}
            g2 = do.cpu().numpy().view(EXT_RESULT_DTYPE)[:s2]
            c2["bitexact_sample"] = f"{int(np.sum(g2 == e2))}/{s2}"
        out["config2"] = c2
        del db, dt, do, do2
        torch.cuda.empty_cache()

    # ---- config 3: 2M mate-rescue local SW (host entry point)
    if want("config3"):
        wl3 = W.config3(n=args.c3_pairs)
        eng.upload_reference(wl3.ref.pac, wl3.ref.n)
        # Inputs and results in pinned host memory (allocated once), as the
        # headline's end-to-end leg.
        pb3 = torch.from_numpy(wl3.bases).pin_memory().numpy()
        pt3 = torch.from_numpy(wl3.tasks.view(np.uint8)).pin_memory().numpy().view(wl3.tasks.dtype)
        po3 = torch.empty(len(wl3.tasks) * LOCAL_RESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy() \
            .view(LOCAL_RESULT_DTYPE)
        eng.local_batch(sc, pb3, pt3[:1000], out=po3)
        t0 = time.perf_counter()
        r3 = eng.local_batch(sc, pb3, pt3, out=po3)
        e2e3 = time.perf_counter() - t0
        ms3, cells3 = eng.last_batch_stats()
        c3 = {"pairs": len(wl3.tasks), "kernel_ms": ms3, "rescues_per_s": len(wl3.tasks) / ms3 * 1e3,
              "buffers": "pinned host memory (bases, tasks, results; allocated once)",
              "e2e_rescues_per_s": len(wl3.tasks) / e2e3, "gcups": cells3 / ms3 / 1e6,
              "hits": int(np.sum(r3["score"] >= 19))}
        if cpu_on:
            s3 = 20_000
            t0 = time.perf_counter()
            e3, _ = oracle.local_batch(sc, wl3.bases, wl3.tasks[:s3], pac=wl3.ref.pac, ref_bases=wl3.ref.n, n_threads=threads)
            c3["cpu_baseline"] = {"value": s3 / (time.perf_counter() - t0), "unit": "rescues/s", "cores": threads,
                                  "kind": "port", "sample": f"first {s3} pairs"}
            c3["bitexact_sample"] = f"{int(np.sum(r3[:s3] == e3))}/{s3}"
        out["config3"] = c3

    # ---- config 3 rescue driver: MateRescue.rescue over 1M mates (swb_mate_rescue)
    if want("config3_rescue_driver"):
        wr = W.config3_jobs(n=args.c3_jobs, ref_len=args.ref_len)
        eng.upload_reference(wr.ref.pac, wr.ref.n)
        rargs = (wr.bases, wr.jobs, wr.templates, wr.mate_regions, wr.stats, wr.primary, wr.contig_offsets,
                 wr.contig_lengths, wr.ref.n)
        eng.mate_rescue(sc, *rargs)
        times = []
        for _ in range(3):
            t0 = time.perf_counter()
            gr, gn, gc = eng.mate_rescue(sc, *rargs)
            times.append(time.perf_counter() - t0)
        e2er = float(np.median(times))
        msr, cellsr = eng.last_batch_stats()
        cr = {"mates": len(wr.jobs), "templates": len(wr.templates), "local_alignments": int(gc.sum()),
              "rescued": int(gn.sum()), "mates_per_s": len(wr.jobs) / e2er, "wall_ms": e2er * 1e3,
              "device_ms": msr, "gcups_device": cellsr / msr / 1e6 if msr else None, "workload": wr.name}
        if cpu_on:
            sr = 20_000
            t0 = time.perf_counter()
            er, en, ec, _ = oracle.mate_rescue_batch(sc, wr.bases, wr.ref.pac, wr.ref.n, wr.jobs[:sr], wr.templates,
                                                     wr.mate_regions, wr.stats, wr.primary, wr.contig_offsets,
                                                     wr.contig_lengths, n_threads=threads)
            cr["cpu_baseline"] = {"value": sr / (time.perf_counter() - t0), "unit": "mates/s", "cores": threads,
                                  "kind": "port", "sample": f"first {sr} mates"}
            same = bool(np.array_equal(gn[:sr], en) and np.array_equal(gc[:sr], ec))
            for j in range(sr):
                o = 4 * int(wr.jobs["tmpl_off"][j])
                if not np.array_equal(gr[o:o + int(en[j])], er[o:o + int(en[j])]):
                    same = False
                    break
            cr["bitexact_sample"] = f"{sr} mates: {'all equal' if same else 'DIFFERENT'}"
        out["config3_rescue_driver"] = cr
        del wr

    # ---- config 1 NW + CIGAR stage (CIGARGenerator.generate through swb_cigar_batch)
    if want("config1_nw_cigar"):
        wl1 = W.config1(n_reads=args.nw_reads, ref_len=args.ref_len)
        eng.upload_reference(wl1.ref.pac, wl1.ref.n)
        info = wl1.read_info
        ct = np.zeros(len(info), CIGAR_TASK_DTYPE)
        L = wl1.read_len
        ct["q_off"] = np.arange(len(info), dtype=np.uint64) * L
        ct["t_off"] = info[:, 0].astype(np.uint64)
        ct["qlen"] = L
        ct["rlen"] = np.minimum(info[:, 1] - info[:, 0], 10_000)
        ct["qb"] = 0
        ct["qe"] = L
        ct["read_len"] = L
        ct["true_score"] = L - info[:, 2] * 5 - info[:, 3] * 2
        ct["initial_w"] = 100
        ct["ref_pos"] = info[:, 0]
        ct["flags"] = 0x8
        # Inputs in pinned host memory, as the headline's end-to-end leg (the
        # call then copies them straight to the device).
        pb1 = torch.from_numpy(wl1.bases).pin_memory().numpy()
        pct = torch.from_numpy(ct.view(np.uint8)).pin_memory().numpy().view(CIGAR_TASK_DTYPE)
        # Outputs in pinned host memory too (allocated once, sized by the
        # library's worst-case rule): the device writes them directly.
        ccap1, mcap1 = eng.cigar_caps(ct)
        pout1 = (torch.empty(len(ct) * CIGAR_RESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy()
                 .view(CIGAR_RESULT_DTYPE),
                 torch.empty(ccap1, dtype=torch.int32).pin_memory().numpy().view(np.uint32),
                 torch.empty(mcap1, dtype=torch.uint8).pin_memory().numpy())
        eng.cigar_batch_raw(sc, pb1, pct, out=pout1)
        times = []
        for _ in range(3):
            eng.profile(True)
            eng.profile_reset()
            t0 = time.perf_counter()
            cres, ccig, cmd = eng.cigar_batch_raw(sc, pb1, pct, out=pout1)
            times.append(time.perf_counter() - t0)
            ms1, cells1 = eng.last_batch_stats()
            prof1 = eng.profile_read()
            eng.profile(False)
        e2e1 = float(np.median(times))
        n_dp = int(cres["used_dp"].sum())
        nw_ms = prof1.get("global_nw_traceback", (0, 0.0))[1]
        c1 = {"reads": len(ct), "dp_alignments": n_dp, "cigars_per_s": len(ct) / e2e1, "wall_ms": e2e1 * 1e3,
              "inputs": "pinned host memory (reads and tasks; results, CIGAR and MD buffers allocated once)",
              "device_ms": ms1, "nw_kernel_ms": nw_ms, "nw_gcups": cells1 / nw_ms / 1e6 if nw_ms else None,
              "nw_alignments_per_s": n_dp / nw_ms * 1e3 if nw_ms else None,
              "kernels": {k: {"launches": v[0], "ms": v[1]} for k, v in prof1.items()}}
        if cpu_on:
            s1 = min(len(ct), 200_000)
            t0 = time.perf_counter()
            eres, ecig, emd, _ = oracle.cigar_batch(sc, wl1.bases, ct[:s1], pac=wl1.ref.pac, n_threads=threads)
            dt1 = time.perf_counter() - t0
            ok = 0
            for k in range(s1):
                g, e = cres[k], eres[k]
                o, n, mo, ml = int(g["cigar_off"]), int(g["n_cigar"]), int(g["md_off"]), int(g["md_len"])
                eo, en, emo, eml = int(e["cigar_off"]), int(e["n_cigar"]), int(e["md_off"]), int(e["md_len"])
                ok += (n == en and ml == eml and (g["score"], g["nm"], g["pos"], g["used_dp"]) ==
                       (e["score"], e["nm"], e["pos"], e["used_dp"]) and np.array_equal(ccig[o:o + n], ecig[eo:eo + en])
                       and np.array_equal(cmd[mo:mo + ml], emd[emo:emo + eml]))
            c1["cpu_baseline"] = {"value": s1 / dt1, "unit": "cigars/s", "cores": threads, "kind": "port",
                                  "sample": f"first {s1} of {len(ct)} reads, CIGARGenerator.generate restated "
                                            f"(orc_cigar_batch), {threads} threads, {dt1:.1f} s"}
            c1["bitexact_sample"] = f"{ok}/{s1}"
        out["config1_nw_cigar"] = c1

    # ---- config 5: ExtensionAligner.extend over 1M seed chains (swb_extend_chains)
    if want("config5_extend_chains"):
        wl5 = W.config5(n_reads=args.c5_chains, ref_len=args.ref_len)
        eng.upload_reference(wl5.ref.pac, wl5.ref.n)
        # Inputs and outputs in pinned host memory (allocated once), as the
        # headline's end-to-end leg: the device reads and writes them directly.
        pb5 = torch.from_numpy(wl5.bases).pin_memory().numpy()
        ps5 = torch.from_numpy(wl5.seeds.view(np.uint8)).pin_memory().numpy().view(wl5.seeds.dtype)
        pc5 = torch.from_numpy(wl5.chains.view(np.uint8)).pin_memory().numpy().view(wl5.chains.dtype)
        po5 = (torch.empty(max(len(wl5.seeds), 1) * REGION_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy()
               .view(REGION_DTYPE),
               torch.empty(max(len(wl5.chains), 1), dtype=torch.int32).pin_memory().numpy().view(np.uint32))
        eng.extend_chains(sc, pb5, ps5, pc5, wl5.ref.n, out=po5)
        times = []
        for _ in range(3):
            t0 = time.perf_counter()
            g5, n5, rounds5 = eng.extend_chains(sc, pb5, ps5, pc5, wl5.ref.n, out=po5)
            times.append(time.perf_counter() - t0)
        e2e5 = float(np.median(times))
        _, cells5 = eng.last_batch_stats()
        c5 = {"chains": len(wl5.chains), "seeds": len(wl5.seeds), "regions": int(n5.sum()), "rounds": rounds5,
              "chains_per_s": len(wl5.chains) / e2e5, "gcups_wall": cells5 / e2e5 / 1e9,
              "buffers": "pinned host memory (bases, seeds, chains, regions, counts; allocated once)"}
        if cpu_on:
            s5 = 100_000
            t0 = time.perf_counter()
            e5, en5, _ = oracle.extend_batch(sc, wl5.bases, wl5.ref.pac, wl5.ref.n, wl5.seeds, wl5.chains[:s5],
                                             n_threads=threads)
            c5["cpu_baseline"] = {"value": s5 / (time.perf_counter() - t0), "unit": "chains/s", "cores": threads,
                                  "kind": "port", "sample": f"first {s5} chains"}
            ok = int(np.array_equal(n5[:s5], en5))
            last = int(wl5.chains["seed_off"][s5 - 1] + en5[-1])
            mask = np.zeros(last, bool)
            for so, n in zip(wl5.chains["seed_off"][:s5], en5):
                mask[so:so + n] = True
            same = int(np.sum(g5[:last][mask] == e5[:last][mask]))
            c5["bitexact_sample"] = f"{same}/{int(mask.sum())} regions, counts equal: {bool(ok)}"
        out["config5_extend_chains"] = c5
        del wl5, g5

    # ---- seeding: SMEMFinder.findAllSMEMs over the config-1 reads (swb_smem_batch)
    if want("seeding"):
        wl6 = W.config1(n_reads=args.seed_reads, ref_len=args.ref_len)
        t0 = time.perf_counter()
        fm = W.fm_index(wl6.ref.codes, device=f"cuda:{dev.index or 0}")
        build_s = time.perf_counter() - t0
        torch.cuda.empty_cache()
        eng.upload_bwt(fm.cp, fm.count, fm.length, fm.sentinel)
        nr = args.seed_reads
        L = wl6.read_len
        off6 = np.arange(nr, dtype=np.uint64) * L
        len6 = np.full(nr, L, np.int32)
        cap6 = 64
        # Phases 1 and 1.25 of alignReadPhase1to3: findAllSMEMs, then internal
        # re-seeding (split length Int(Float(19) * 1.5 + 0.499) = 28, split width 10).
        split6 = oracle.split_len_of(19, 1.5)
        # One call with library-sized outputs sizes the pinned output buffers;
        # the timed calls read pinned reads and write pinned outputs directly.
        _, n0, _ = eng.smem_batch(wl6.bases, off6, len6, 19, cap_per_read=cap6, split_len=split6)
        tot6 = int(n0.sum())
        pb6 = torch.from_numpy(wl6.bases).pin_memory().numpy()
        poff6 = torch.from_numpy(off6.view(np.uint8)).pin_memory().numpy().view(np.uint64)
        plen6 = torch.from_numpy(len6.view(np.uint8)).pin_memory().numpy().view(np.int32)
        pout6 = (torch.empty((tot6 + 1024) * SMEM_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy()
                 .view(SMEM_DTYPE),
                 torch.empty(nr, dtype=torch.int32).pin_memory().numpy().view(np.uint32),
                 torch.empty(nr * 8, dtype=torch.uint8).pin_memory().numpy().view(np.uint64))
        eng.smem_batch(pb6, poff6, plen6, 19, cap_per_read=cap6, split_len=split6, out=pout6)
        times = []
        for _ in range(3):
            t0 = time.perf_counter()
            sm6, n6, o6 = eng.smem_batch(pb6, poff6, plen6, 19, cap_per_read=cap6, split_len=split6, out=pout6)
            times.append(time.perf_counter() - t0)
        e2e6 = float(np.median(times))
        ms6, exts6 = eng.last_batch_stats()
        # Bytes the rank queries read: one or two 64-byte checkpoints per
        # backward extension, counted as 96 bytes (1.5 checkpoints) each.
        c6 = {"reads": nr, "read_len": L, "smems": int(n6.sum()), "kernel_ms": ms6,
              "buffers": "pinned host memory (reads, offsets, lengths, SMEMs, counts, offsets; allocated once)",
              "reads_per_s_kernel": nr / ms6 * 1e3, "reads_per_s_e2e": nr / e2e6,
              "smems_per_s_kernel": float(n6.sum()) / ms6 * 1e3,
              "backward_extensions": int(exts6), "backward_ext_per_s": exts6 / ms6 * 1e3,
              "index": f"{wl6.ref.n // 10**6} Mbp forward strand + reverse complement, {fm.cp.size} checkpoints "
                       f"({fm.cp.nbytes / 1e6:.0f} MB resident, larger than L2), built in {build_s:.1f} s",
              "approx_checkpoint_gbs": exts6 * 96 / ms6 / 1e6}
        if cpu_on:
            s6 = min(nr, 100_000)
            t0 = time.perf_counter()
            e6, en6, _ = oracle.smem_batch(oracle.FMIndex(fm.cp, fm.count, fm.length, fm.sentinel), wl6.bases,
                                           off6[:s6], len6[:s6], 19, cap=cap6, n_threads=threads,
                                           split_len=split6, split_width=10)
            dt6 = time.perf_counter() - t0
            c6["cpu_baseline"] = {"value": s6 / dt6, "unit": "reads/s", "cores": threads, "kind": "port",
                                  "sample": f"first {s6} reads, SMEMFinder.findAllSMEMs + internalReseed restated, "
                                            f"{threads} threads, "
                                            f"{dt6:.1f} s"}
            same6 = bool(np.array_equal(n6[:s6], en6))
            for r in range(s6):
                if not np.array_equal(sm6[o6[r]: o6[r] + n6[r]], e6[r * cap6: r * cap6 + en6[r]]):
                    same6 = False
                    break
            c6["bitexact_sample"] = f"{s6} reads: {'all equal' if same6 else 'DIFFERENT'}"
        out["seeding"] = c6
        del wl6, fm

    # ---- config 4: serving, Poisson 200 req/s, 1 Gbp resident reference
    if want("config4"):
        from swiftbwa_b200 import serving as S
        ref4 = W.reference(W.SEED_BASE + 4, args.c4_ref_len)
        eng.upload_reference(ref4.pac, ref4.n)
        pool = W.uneven(ref4, W.SEED_BASE + 4 + 1, args.c4_pool, name="config4 pool")
        tune4 = None if args.no_tune else eng.tune_ext_bins(sc, pool.bases, pool.tasks[: args.tune_sample or None])
        # The serving process keeps its read chunks in pinned memory, so requests
        # are zero-copy views of the pool.
        pb = torch.from_numpy(pool.bases).pin_memory().numpy()
        pt = torch.from_numpy(pool.tasks.view(np.uint8)).pin_memory().numpy().view(pool.tasks.dtype)
        po = torch.empty(len(pool.tasks) * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy().view(EXT_RESULT_DTYPE)
        reqs = S.request_stream(W.SEED_BASE + 4 + 2, len(pool.tasks), rate=200.0, duration=args.serve_seconds)
        srv = S.Server(eng, sc, arena_bytes=1 << 30, max_wave_tasks=args.c4_wave, latency_cells=args.c4_latency_cells)
        _warm_server(S, srv, pb, pt, po, reqs)
        res, span = S.run_pool_stream(srv, pb, pt, po, reqs, open_loop=True)
        st = srv.stats()
        srv.stop()
        # Served results of the first requests (about 200k tasks) against the oracle.
        chk, tot = [], 0
        for r in reqs:
            if tot >= 200_000:
                break
            chk.append(r)
            tot += r.hi - r.lo
        same4 = 0
        t0 = time.perf_counter()
        for r in chk:
            e4, _ = oracle.ext_batch(sc, pool.bases, pool.tasks[r.lo:r.hi], pac=ref4.pac, ref_bases=ref4.n,
                                     n_threads=threads)
            same4 += int(np.sum(po[r.lo:r.hi] == e4))
        dt4 = time.perf_counter() - t0
        lat = [l for _, l in res]
        mid = [l for n, l in res if 50_000 <= n <= 200_000]
        near100k = [l for n, l in res if 70_000 <= n <= 140_000]
        c4 = {"requests": len(reqs), "tasks": int(sum(n for n, _ in res)), "offered_req_per_s": 200.0,
              "ext_per_s": sum(n for n, _ in res) / span, "p50_ms": _pct(lat, 50) * 1e3, "p99_ms": _pct(lat, 99) * 1e3,
              "p50_ms_50k_200k": _pct(mid, 50) * 1e3 if mid else None,
              "p99_ms_50k_200k": _pct(mid, 99) * 1e3 if mid else None, "n_50k_200k": len(mid),
              "p50_ms_70k_140k": _pct(near100k, 50) * 1e3 if near100k else None,
              "p99_ms_70k_140k": _pct(near100k, 99) * 1e3 if near100k else None, "n_70k_140k": len(near100k),
              "waves": st["waves"], "wave_tasks": args.c4_wave, "latency_cells": args.c4_latency_cells, "ext_bins": eng.ext_bins(), "ext_bins_tuning": tune4, "wave_device_ms_sum": st["busy_ms"], "span_s": span,
              "stream": "Poisson 200 req/s, sizes log-uniform 1k-1M tasks, qlen log-uniform 30-250, w 10-100, h0 19-60, "
                        "1 Gbp resident 2-bit reference",
              "bitexact_sample": f"{same4}/{tot} served results of the first {len(chk)} requests equal the oracle"}
        if cpu_on:
            c4["cpu_baseline"] = {"value": tot / dt4, "unit": "ext/s", "cores": threads, "kind": "port",
                                  "sample": f"the first {len(chk)} requests of the stream ({tot} tasks), "
                                            f"BandedSWScalar.align restated, {threads} threads, {dt4:.1f} s"}
        # saturation: the same size distribution submitted at once, served vs plain
        sat = S.request_stream(W.SEED_BASE + 4 + 3, len(pool.tasks), rate=1e6, duration=args.sat_requests / 1e6)
        for mode, plain in (("served", 0), ("plain_batching", 1), ("plain_kernel", 2)):
            srv = S.Server(eng, sc, arena_bytes=1 << 30, max_wave_tasks=args.c4_wave if plain == 0 else 1 << 20,
                           plain=plain, latency_cells=args.c4_latency_cells if plain == 0 else 0)
            _warm_server(S, srv, pb, pt, po, sat)
            r_, span_ = S.run_pool_stream(srv, pb, pt, po, sat, open_loop=False)
            srv.stop()
            c4[f"saturation_{mode}_ext_per_s"] = sum(n for n, _ in r_) / span_
            c4[f"saturation_{mode}_p99_ms"] = _pct([l for _, l in r_], 99) * 1e3
        c4["saturation_requests"] = len(sat)
        c4["served_over_plain_batching"] = c4["saturation_served_ext_per_s"] / c4["saturation_plain_batching_ext_per_s"]
        c4["served_over_plain_kernel"] = c4["saturation_served_ext_per_s"] / c4["saturation_plain_kernel_ext_per_s"]
        out["config4"] = c4
    return out


# --------------------------------------------------------- reference arm
def run_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0:
        return
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.abi import Scoring
    from oracle import oracle
    sc = Scoring.default()
    wl = W.config1(rank=0, n_reads=args.n_reads, ref_len=args.ref_len)
    threads = os.cpu_count() or 1
    n = len(wl.tasks)
    probe = min(n, 20_000)
    t0 = time.perf_counter()
    oracle.ext_batch(sc, wl.bases, wl.tasks[:probe], pac=wl.ref.pac, ref_bases=wl.ref.n, n_threads=threads)
    rate = probe / max(time.perf_counter() - t0, 1e-6)
    total_budget = 150.0
    s = int(min(n, max(probe, rate * total_budget / max(args.steps + args.warmup, 1))))
    times, cells_tot = [], 0
    for it in range(args.warmup + args.steps):
        lo = (it * s) % max(n - s, 1)
        t0 = time.perf_counter()
        _, cells = oracle.ext_batch(sc, wl.bases, wl.tasks[lo:lo + s], pac=wl.ref.pac, ref_bases=wl.ref.n,
                                    n_threads=threads)
        dt = time.perf_counter() - t0
        if it >= args.warmup:
            times.append(dt)
            cells_tot += cells
    tot = sum(times)
    value = s * len(times) / tot
    line = {"impl": "reference", "metric": "extensions/s (bit-exact banded SW extension, config 1)",
            "value": value, "unit": "ext/s", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * tot / len(times), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32", "data": "synthetic (seeded config-1 generator)",
            "config": {"workload": wl.name, "sample_tasks_per_step": s},
            "gcups": cells_tot / tot / 1e9,
            "cpu_baseline": {"value": value, "unit": "ext/s", "cores": threads, "kind": "port",
                             "sample": f"{s} of {n} config-1 tasks per step, C++ restatement of BandedSWScalar.align, {threads} threads"},
            "e2e": {"value": value, "unit": "ext/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# ----------------------------------------------------------------- our arm
def run_ours(args):
    ws, rank, local = dist_env()
    import torch
    dist = None
    if ws > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=600))
    else:
        torch.cuda.set_device(local)
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.abi import EXT_RESULT_DTYPE, Scoring
    from swiftbwa_b200.alignment import Engine
    from swiftbwa_b200.build import build
    build()

    sc = Scoring.default()
    if args.suite_only:
        if rank == 0:
            eng = Engine(local)
            only = {x.strip() for x in args.suite_only.split(",") if x.strip()}
            suite = secondary_suite(eng, sc, args, torch.device("cuda", local), torch, cpu_on=not args.no_cpu,
                                    only=only)
            print(json.dumps({"suite_only": sorted(only), "configs": suite}), flush=True)
        return
    t_gen = time.perf_counter()
    wl = W.config1(rank=rank, n_reads=args.n_reads, ref_len=args.ref_len)
    t_gen = time.perf_counter() - t_gen
    n = len(wl.tasks)
    eng = Engine(local)
    eng.upload_reference(wl.ref.pac, wl.ref.n)
    # Length classes of the bins, autotuned on a sample of this workload
    # before any timing (one-time setup, like a library's algorithm search).
    tune1 = None if args.no_tune else eng.tune_ext_bins(sc, wl.bases, wl.tasks[: args.tune_sample or None])
    bins1 = eng.ext_bins()   # the classes the timed passes use (the suite re-tunes later)
    probe_clk = ClockSampler(local)
    probe_clk.start()
    time.sleep(0.3)
    alu_peak = eng.int_alu_peak()
    alu16_peak = eng.int16x2_alu_peak()
    probe_clk = probe_clk.stop()

    # HBM-resident inputs (torch only allocates; the library computes).
    dev = torch.device("cuda", local)
    d_bases = torch.from_numpy(wl.bases).to(dev)
    d_tasks = torch.from_numpy(wl.tasks.view(np.uint8)).to(dev)
    d_out = torch.empty(n * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8, device=dev)
    # A dedicated stream: the library's kernels and the timing events both go
    # on it (a NULL handle would select the library's own context stream).
    stream = torch.cuda.Stream(dev)
    torch.cuda.synchronize()

    def step():
        eng.ext_batch_device(sc, d_bases.data_ptr(), d_tasks.data_ptr(), n, d_out.data_ptr(), stream.cuda_stream)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    launches0 = eng.kernel_launches()
    clocks = ClockSampler(local)
    clocks.start()
    time.sleep(0.3)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    w0 = time.perf_counter()
    e0.record(stream)
    for _ in range(args.steps):
        step()
    e1.record(stream)
    torch.cuda.synchronize()
    wall_ms = (time.perf_counter() - w0) * 1e3 / args.steps
    if dist:
        dist.barrier()
    ms = e0.elapsed_time(e1) / args.steps
    clk = clocks.stop()
    launches = eng.kernel_launches() - launches0
    ms_max = max_over_ranks(ms, dist, dev)
    gpu_out = d_out.cpu().numpy().view(EXT_RESULT_DTYPE)
    # The kernel breakdown and the reference's cell count, outside the timed
    # steps: under profiling the kernels compute every row the reference does,
    # so these passes take longer than the timed ones.
    prof_steps = 2
    eng.profile(True)
    eng.profile_reset()
    for _ in range(prof_steps):
        step()
    prof = eng.profile_read()
    eng.profile(False)
    assert np.array_equal(d_out.cpu().numpy().view(EXT_RESULT_DTYPE), gpu_out), "profiled and timed passes disagree"

    cells_step = sum(v[2] for v in prof.values()) / prof_steps
    # The length bins run concurrently on their own streams, so the unit the
    # roofline measures is a whole step: keys, sort and bins.  Its cells are those
    # that the timed form computes: the counters of one step as timed and one that
    # computes every row, less the latter's.
    eng.profile_reset()
    step()
    eng.profile(True)
    step()
    both = eng.profile_read()
    eng.profile(False)
    cells_timed = sum(v[2] for v in both.values()) - cells_step
    dom_name = "one step (ext_keys, radix sort, bin_bounds, ext_fast_q32..q256 + ext_big_i32, concurrent bins)"
    achieved = cells_timed * OPS_PER_CELL_EXT / (ms_max * 1e-3)
    # The profiled pass with every row, fork to join on the launching stream.
    pass_launches, pass_ms, _ = prof["ext_pass"]
    bin_cells = sum(v[2] for k, v in prof.items() if k.startswith("ext_"))
    every_row = (bin_cells / pass_launches) * OPS_PER_CELL_EXT / (pass_ms / pass_launches * 1e-3)
    step_ms_sum = sum(v[1] for k, v in prof.items() if k in ("ext_keys", "cub_radix_sort", "bin_bounds", "ext_pass"))
    kernels = {k: {"launches": v[0], "ms_per_step": v[1] / prof_steps,
                   "share_of_step": (v[1] / step_ms_sum) if k in ("ext_keys", "cub_radix_sort", "bin_bounds", "ext_pass") else None,
                   "cells_per_step": v[2] / prof_steps,
                   "gcups_in_own_window": (v[2] / (v[1] * 1e-3) / 1e9) if v[2] else None} for k, v in prof.items()}

    # End to end through the host entry point, pinned host buffers.
    e2e = None
    if not args.no_e2e:
        hb = torch.from_numpy(wl.bases).pin_memory().numpy()
        ht = torch.from_numpy(wl.tasks.view(np.uint8)).pin_memory().numpy().view(wl.tasks.dtype)
        ho = torch.empty(n * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy().view(EXT_RESULT_DTYPE)
        eng.ext_batch(sc, hb, ht, out=ho)
        if dist:
            dist.barrier()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            eng.ext_batch(sc, hb, ht, out=ho)
        wall = max_over_ranks((time.perf_counter() - t0) / args.steps, dist, dev)
        assert np.array_equal(ho, gpu_out), "host and device entry points disagree"
        e2e = {"value": whole_job_rate(n, ws, wall), "unit": "ext/s", "h2d_bytes_per_step": int(hb.nbytes + ht.nbytes),
               "d2h_bytes_per_step": int(ho.nbytes), "ms_per_step": wall * 1e3}

    cpu = None
    if rank == 0 and ws == 1 and not args.no_cpu:
        cpu = cpu_baseline(wl, sc, args.cpu_seconds, gpu_out)
    suite = None
    if rank == 0 and ws == 1 and not args.no_suite:
        del d_bases, d_tasks, d_out
        torch.cuda.empty_cache()
        suite = secondary_suite(eng, sc, args, dev, torch, cpu_on=not args.no_cpu)

    if rank == 0:
        line = {
            "metric": "extensions/s (bit-exact banded SW extension, config 1)",
            "value": whole_job_rate(n, ws, ms_max * 1e-3), "unit": "ext/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_max, "wall_ms_per_step": wall_ms,
            "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32",
            "data": "synthetic (seeded config-1 generator: reads, errors, tandem repeats)",
            "config": {"workload": wl.name, "tasks_per_gpu": n, "reads_per_gpu": args.n_reads, "read_len": 150,
                       "ref_bases": wl.ref.n, "w": 100, "h0": 19, "end_bonus": 5,
                       "l2": f"inputs larger than L2 ({(wl.bases.nbytes + wl.tasks.nbytes) / 1e6:.0f} MB read per step)",
                       "parallelism": f"replicas x{ws} (task shards, no collective)",
                       "ext_bins": bins1, "ext_bins_tuning": tune1},
            "gcups": cells_step * ws / (ms_max * 1e-3) / 1e9,   # the reference's cells, rows left out included
            "cells_per_step_per_gpu": cells_step,
            "cells_computed_per_step_per_gpu": cells_timed,
            "roofline": {"bound": "alu", "kernel": dom_name, "achieved": achieved / 1e12,
                         "avg_launch_ms": ms_max,
                         "every_row_pass": {"ms": pass_ms / pass_launches, "achieved": every_row / 1e12,
                                            "frac": every_row / alu16_peak},
                         "peak": alu16_peak / 1e12,
                         "unit": "T int16 lane ops/s (13 ops per DP cell; peak: packed 16-bit DPX add/max probe)",
                         "frac": achieved / alu16_peak, "traffic": traffic_per_launch("ext_pass"),
                         "ops_per_cell": OPS_PER_CELL_EXT,
                         "peak_source": "measured in this run on this GPU: swb_int16x2_alu_peak (s16x2 viaddmax "
                                        "chains, 2 lanes x add+max per instruction); MEASURED_PEAKS.json has no "
                                        "integer figure",
                         "peak_sm_mhz": probe_clk.get("sm_mhz"), "achieved_sm_mhz": clk.get("sm_mhz"),
                         "int32_peak": alu_peak / 1e12, "int32_frac": achieved / alu_peak,
                         "int32_unit": "T int32 ops/s (s32 viaddmax probe, swb_int_alu_peak)"},
            "kernels": kernels,
            "gpu_launches": int(launches),
            "clocks": clk,
            "e2e": e2e,
            "cpu_baseline": cpu,
            "configs": suite,
            "gen_seconds": t_gen,
        }
        print(json.dumps(line), flush=True)
    eng.close()
    if dist:
        dist.destroy_process_group()


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
