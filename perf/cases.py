"""Performance cases of the library's public entry points.

Each case is one call (or one burst of requests) that a short-read aligner
makes: single alignments, seed extension of small, ordinary and large batches
(HBM-resident and from host memory), NW + CIGAR, local SW, mate rescue, whole
seed chains, SMEM seeding and the request server.  Inputs are the seeded
synthetic reads of swiftbwa_b200.workloads off one fixed 100 Mbp genome (2 %
of it tandem repeats), which stays resident with its FM index, as an
aligner's reference does; a seed changes the reads, never the genome.  One
Engine serves the process (alignment.default_engine()), host buffers are
pinned and allocated once, and the default scoring is used.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the caller holds before the call
  run(state)           one pass through the public entry points
  work(case)           bytes and integer operations of one pass
  exact(case, seed)    None: every output is a whole number
"""
import math

import numpy as np
import torch

from swiftbwa_b200 import workloads as W
from swiftbwa_b200.abi import (CIGAR_RESULT_DTYPE, CIGAR_TASK_DTYPE, EXT_RESULT_DTYPE, LOCAL_RESULT_DTYPE,
                               LOCAL_TASK_DTYPE, REGION_DTYPE, SMEM_DTYPE, SWB_T_FROM_REF, Scoring)
from swiftbwa_b200.alignment import default_engine
from swiftbwa_b200.serving import Server

GENOME = 100_000_000
MIN_SEED = 19
SPLIT_LEN = 28          # re-seeding length of the default scoring: Int(19 * 1.5 + 0.499)
SMEMS_PER_READ = 32     # pinned output entries per read
CONTIGS = 24

# Read error rates: the reads of configs 0, 1 and 5 (1 % substitutions, 0.1 %
# indels, 0.5 % N); the uneven and rescue workloads have 2 % substitutions.
LISTED = [
    # One alignment of each kind through the reference's single-call signatures.
    dict(name="single_calls", kind="single", qlen=100, extra=100, window=700),
    # A small batch from host memory: right extensions of 100 bp reads (config 0).
    dict(name="ext_host_10k", kind="ext_host", n=10_000, read_len=100, sides=1),
    # A serving-wave-sized batch in HBM with queries of 30-250 bases and bands of 10-100 (config 2).
    dict(name="ext_device_131k", kind="ext_uneven", n=131_072, qmin=30, qmax=250, wmin=10, wmax=100),
    # Left and right extensions of 1M reads of 150 bp in HBM (config 1).
    dict(name="ext_device_2m", kind="ext_reads", n=2_000_000, read_len=150),
    # A large uneven batch in HBM (config 2), above the size where bands become rings.
    dict(name="ext_device_5m", kind="ext_uneven", n=5_000_000, qmin=30, qmax=250, wmin=10, wmax=100),
    # The same work as ext_device_2m end to end from pinned host memory, half the size.
    dict(name="ext_host_1m", kind="ext_host", n=1_000_000, read_len=150, sides=2),
    # NW + CIGAR + MD of a chunk of aligned reads.
    dict(name="cigar_100k", kind="cigar", n=100_000, read_len=150),
    # Mate-rescue local alignments: 150 bp mates against 700 bp windows (config 3).
    dict(name="local_50k", kind="local", n=50_000, qlen=150, window=700),
    # The rescue driver: candidate windows, local alignments and regions of 50k mates.
    dict(name="rescue_50k", kind="rescue", n=50_000, read_len=150),
    # ExtensionAligner.extend over the seed chains of a chunk of reads (config 5).
    dict(name="chains_200k", kind="chains", n=200_000, read_len=150),
    # SMEM seeding with internal re-seeding of a chunk of reads.
    dict(name="seed_100k", kind="seed", n=100_000, read_len=150),
    # A burst of 16 concurrent extension requests of 1k-100k tasks through the request server (config 4).
    dict(name="serve_16", kind="serve", requests=16, lo=1_000, hi=100_000),
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "ext_host", "ext_host", "ext_uneven", "ext_uneven", "ext_reads", "cigar", "local",
                       "local", "rescue", "chains", "seed", "serve"])
    read_len = rng.choice([100, 101, 125, 150, 151, 250])
    if kind == "single":
        return dict(kind=kind, qlen=rng.randint(20, 250), extra=rng.randint(1, 120), window=rng.randint(300, 1000))
    if kind == "ext_host":
        return dict(kind=kind, n=_log_int(rng, 100, 500_000), read_len=read_len, sides=rng.choice([1, 2]))
    if kind == "ext_reads":
        return dict(kind=kind, n=_log_int(rng, 1_000, 1_000_000), read_len=read_len)
    if kind == "ext_uneven":
        qmin = rng.randint(20, 60)
        qmax = rng.choice([rng.randint(100, 250), 250, rng.randint(251, 400)])
        wmin = rng.randint(5, 30)
        return dict(kind=kind, n=_log_int(rng, 1_000, 4_000_000 if qmax <= 250 else 100_000), qmin=qmin, qmax=qmax,
                    wmin=wmin, wmax=rng.randint(wmin + 1, 120))
    if kind == "cigar":
        return dict(kind=kind, n=_log_int(rng, 100, 80_000), read_len=read_len)
    if kind == "local":
        return dict(kind=kind, n=_log_int(rng, 50, 40_000), qlen=rng.choice([36, 75, read_len]),
                    window=rng.randint(400, 900))
    if kind == "rescue":
        return dict(kind=kind, n=_log_int(rng, 1_000, 40_000), read_len=rng.choice([100, 125, 150]))
    if kind == "chains":
        return dict(kind=kind, n=_log_int(rng, 100, 150_000), read_len=read_len)
    if kind == "seed":
        return dict(kind=kind, n=_log_int(rng, 100, 80_000), read_len=rng.choice([75, 100, 125, 150]))
    return dict(kind=kind, requests=rng.randint(2, 24), lo=_log_int(rng, 200, 2_000), hi=_log_int(rng, 4_000, 60_000))


# ----------------------------------------------------------- resident objects
_kept = {}


def _genome():
    if "genome" not in _kept:
        _kept["genome"] = W.reference(W.SEED_BASE + 1, GENOME, tandem_frac=0.02)
        default_engine().upload_reference(_kept["genome"].pac, GENOME)
    return _kept["genome"]


def _index():
    ref = _genome()
    if "index" not in _kept:
        fm = W.fm_index(ref.codes, device="cuda")
        torch.cuda.empty_cache()
        default_engine().upload_bwt(fm.cp, fm.count, fm.length, fm.sentinel)
        _kept["index"] = True


def _server():
    _genome()
    if "server" not in _kept:
        _kept["server"] = Server(default_engine(), Scoring.default(), arena_bytes=1 << 30, max_wave_tasks=131_072)
    return _kept["server"]


def _stream():
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
    return _kept["stream"]


def _pin(a):
    """The array in pinned host memory (contiguous bytes copied once)."""
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.uint8).reshape(-1)).pin_memory().numpy().view(a.dtype)


def _pinned_zeros(n, dtype):
    dtype = np.dtype(dtype)
    t = torch.zeros(max(n, 1) * dtype.itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(dtype)


def _i32(a):
    """Records of 32- and 64-bit fields as rows of int32 words."""
    return a.view(np.int32).reshape(len(a), -1)


def _mixed(seed):
    """The generator's seed: distinct streams for distinct seeds."""
    return (seed * 0x9E3779B97F4A7C15 + 0x5EED) & 0x7FFFFFFFFFFFFFFF


# ------------------------------------------------------------------ prepare
def _read_tasks(seed, n, read_len, sides):
    """Exactly n extension tasks of simulated reads (some reads give fewer
    than `sides` tasks: a seed at either end leaves nothing to extend)."""
    ref = _genome()
    reads = n // sides + n // (12 * sides) + 64
    while True:
        wl = W.ext_from_reads(ref, _mixed(seed), reads, read_len, left=sides == 2, random_seed_pos=sides == 2,
                              tandem_read_frac=0.2 if sides == 2 else 0.0)
        if len(wl.tasks) >= n:
            used = int(wl.tasks["q_off"][n - 1] // read_len + 1) * read_len
            return wl.bases[:used], wl.tasks[:n]
        reads *= 2


def _request_sizes(case):
    k, lo, hi = case["requests"], case["lo"], case["hi"]
    return [int(lo * (hi / lo) ** (i / max(k - 1, 1))) for i in range(k)]


def prepare(case, seed):
    kind = case["kind"]
    ref = _genome()
    st = dict(kind=kind, sc=Scoring.default(), eng=default_engine())
    if kind == "single":
        rng = np.random.default_rng(seed)
        q, extra, win = case["qlen"], case["extra"], case["window"]
        p = int(rng.integers(0, GENOME - q - extra - win))
        t = ref.codes[p:p + q + extra].copy()
        query = t[:q].copy()
        sub = rng.random(q) < 0.02
        query[sub] = (query[sub] + 1 + rng.integers(0, 3, int(sub.sum()))) & 3
        at = int(rng.integers(0, max(win - q, 1)))
        st.update(q=query, t=t, window=ref.codes[max(p - at, 0):max(p - at, 0) + win].copy())
    elif kind == "ext_host":
        b, t = _read_tasks(seed, case["n"], case["read_len"], case["sides"])
        st.update(bases=_pin(b), tasks=_pin(t), out=_pinned_zeros(case["n"], EXT_RESULT_DTYPE))
    elif kind in ("ext_reads", "ext_uneven"):
        if kind == "ext_reads":
            b, t = _read_tasks(seed, case["n"], case["read_len"], 2)
        else:
            wl = W.uneven(ref, _mixed(seed), case["n"], qmin=case["qmin"], qmax=case["qmax"], wmin=case["wmin"],
                          wmax=case["wmax"])
            b, t = wl.bases, wl.tasks
        st.update(n=case["n"], bases=torch.from_numpy(b).cuda(), tasks=torch.from_numpy(t.view(np.uint8)).cuda(),
                  out=torch.zeros(case["n"] * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda"),
                  stream=_stream())
    elif kind == "cigar":
        n, L = case["n"], case["read_len"]
        wl = W.ext_from_reads(ref, _mixed(seed), n, L, tandem_read_frac=0.2)
        info = wl.read_info
        ct = np.zeros(n, CIGAR_TASK_DTYPE)
        ct["q_off"] = np.arange(n, dtype=np.uint64) * L
        ct["t_off"] = info[:, 0]
        ct["qlen"] = ct["qe"] = ct["read_len"] = L
        ct["rlen"] = info[:, 1] - info[:, 0]
        ct["true_score"] = L - info[:, 2] * 5 - info[:, 3] * 2
        ct["initial_w"] = 100
        ct["ref_pos"] = info[:, 0]
        ct["flags"] = SWB_T_FROM_REF
        cig, md = st["eng"].cigar_caps(ct)
        span = 2 * L + 16     # an upper bound of qlen + rlen, the same for every seed
        st.update(bases=_pin(wl.bases), tasks=_pin(ct),
                  out=(_pinned_zeros(n, CIGAR_RESULT_DTYPE), _pinned_zeros(max(cig, n * (span + 2)), np.uint32),
                       _pinned_zeros(max(md, n * (6 * span + 8)), np.uint8)))
    elif kind == "local":
        n, q, win = case["n"], case["qlen"], case["window"]
        bases = np.empty(n * q, np.uint8)
        tasks = np.empty(n, LOCAL_TASK_DTYPE)
        W.lib().swbw_rescue_tasks(_mixed(seed), ref.codes.ctypes.data, ref.n, n, q, win, 400.0, 50.0, 0.02, 0.10,
                                  MIN_SEED, bases.ctypes.data, tasks.ctypes.data)
        st.update(bases=_pin(bases), tasks=_pin(tasks), out=_pinned_zeros(n, LOCAL_RESULT_DTYPE))
    elif kind == "rescue":
        n = case["n"]
        rj = W.rescue_jobs(ref, seed, n, case["read_len"], n_contigs=CONTIGS)
        slots = int(2.1 * n) + 128          # template entries, the same for every seed
        tmpl = np.zeros(max(slots, len(rj.templates)), rj.templates.dtype)
        tmpl[:len(rj.templates)] = rj.templates
        # Output entry -> its job and its place among the job's entries.
        job = np.repeat(np.arange(n), 4 * rj.jobs["n_tmpl"].astype(np.int64))
        first = np.repeat(4 * rj.jobs["tmpl_off"].astype(np.int64), 4 * rj.jobs["n_tmpl"].astype(np.int64))
        st.update(args=(rj.bases, rj.jobs, tmpl, rj.mate_regions, rj.stats, rj.primary, rj.contig_offsets,
                        rj.contig_lengths, ref.n), job=job, rank=np.arange(len(job)) - first)
    elif kind == "chains":
        wl = W.chains(ref, _mixed(seed), case["n"], case["read_len"])
        st.update(bases=_pin(wl.bases), seeds=_pin(wl.seeds), chains=_pin(wl.chains),
                  out=(_pinned_zeros(7 * case["n"], REGION_DTYPE), _pinned_zeros(case["n"], np.uint32)))
    elif kind == "seed":
        _index()
        n, L = case["n"], case["read_len"]
        wl = W.ext_from_reads(ref, _mixed(seed), n, L, tandem_read_frac=0.2)
        st.update(bases=_pin(wl.bases), off=_pin(np.arange(n, dtype=np.uint64) * L), lens=_pin(np.full(n, L, np.int32)),
                  out=(_pinned_zeros(n * SMEMS_PER_READ, SMEM_DTYPE), _pinned_zeros(n, np.uint32),
                       _pinned_zeros(n, np.uint64)))
    else:
        reqs = []
        for k, n in enumerate(_request_sizes(case)):
            wl = W.uneven(ref, _mixed(seed * 64 + k), n, mix=[100, 150, 250])
            reqs.append((_pin(wl.bases), _pin(wl.tasks), _pinned_zeros(n, EXT_RESULT_DTYPE)))
        st.update(reqs=reqs, server=_server())
    return st


# ---------------------------------------------------------------------- run
def run(st):
    kind, eng, sc = st["kind"], st["eng"], st["sc"]
    if kind == "single":
        e = eng.banded_sw_align(st["q"], st["t"], sc, 100, MIN_SEED, 5)
        g = eng.global_align(st["q"], st["t"][:len(st["q"])], sc, 100)
        loc = eng.local_align(st["q"], st["window"], sc, MIN_SEED)
        return [list(e.as_tuple()), [g.score, *g.cigar], list(loc.as_tuple()) if loc else [0] * 6]
    if kind == "ext_host":
        return _i32(eng.ext_batch(sc, st["bases"], st["tasks"], out=st["out"]))
    if kind in ("ext_reads", "ext_uneven"):
        eng.ext_batch_device(sc, st["bases"].data_ptr(), st["tasks"].data_ptr(), st["n"], st["out"].data_ptr(),
                             st["stream"].cuda_stream)
        return st["out"].view(torch.int32).view(-1, 6)
    if kind == "cigar":
        res, cig, md = eng.cigar_batch_raw(sc, st["bases"], st["tasks"], out=st["out"])
        return [_i32(res), cig, md]
    if kind == "local":
        return _i32(eng.local_batch(sc, st["bases"], st["tasks"], out=st["out"]))
    if kind == "rescue":
        out, n_out, n_cand = eng.mate_rescue(sc, *st["args"])
        rows = _i32(out)
        used = len(st["job"])
        rows[used:] = 0
        rows[:used][st["rank"] >= n_out[st["job"]]] = 0      # entries past a job's regions hold nothing
        return [rows, n_out, n_cand]
    if kind == "chains":
        regions, counts, rounds = eng.extend_chains(sc, st["bases"], st["seeds"], st["chains"], GENOME, out=st["out"])
        return [_i32(regions), counts, rounds]
    if kind == "seed":
        smems, n_out, off = eng.smem_batch(st["bases"], st["off"], st["lens"], MIN_SEED, cap_per_read=64,
                                           split_len=SPLIT_LEN, out=st["out"])
        return [_i32(smems), n_out, off.view(np.int64)]
    tickets = [st["server"].submit(b, t, out=o) for b, t, o in st["reqs"]]
    return [_i32(st["server"].wait(tk)[0]) for tk in tickets]


# --------------------------------------------------------------------- work
def _ext_work(n, q_mean, q_sq, t_mean):
    """40-byte task, query bytes, 2-bit target and 24-byte result; about
    0.75 q^2 band cells of 13 operations (band narrowing leaves that much of
    the matrix on the read workloads)."""
    return n * (64 + q_mean + t_mean / 4), 13 * 0.75 * q_sq * n


def _uneven_work(n, qmin, qmax, w):
    lr = math.log(qmax / qmin)
    q_mean, q_sq = (qmax - qmin) / lr, (qmax ** 2 - qmin ** 2) / (2 * lr)
    return _ext_work(n, q_mean, q_sq, q_mean + w)


def work(case):
    kind = case["kind"]
    if kind == "single":
        q, t, win = case["qlen"], case["qlen"] + case["extra"], case["window"]
        b, f = 3 * q + t + q + win + 100, 13 * 0.75 * q * q + 17 * q * q + 12 * q * win
    elif kind in ("ext_host", "ext_reads"):
        free = case["read_len"] - MIN_SEED
        if case.get("sides", 2) == 2:       # the seed lies anywhere: either side has 0..free bases
            b, f = _ext_work(case["n"], free / 2, free * free / 3, free / 2 + 100)
        else:
            b, f = _ext_work(case["n"], free, free * free, free + 100)
    elif kind == "ext_uneven":
        b, f = _uneven_work(case["n"], case["qmin"], case["qmax"], (case["wmin"] + case["wmax"]) / 2)
    elif kind == "cigar":
        n, L = case["n"], case["read_len"]   # about half of the reads need the DP, 17 operations a cell
        b, f = n * (64 + L + L / 4 + 48 + 8 + 16), 17 * 0.5 * n * L * L
    elif kind == "local":
        n, q, win = case["n"], case["qlen"], case["window"]   # forward pass, then back from the hit's end
        b, f = n * (32 + q + win / 4 + 24), 12 * n * q * win * 1.5
    elif kind == "rescue":
        n, L = case["n"], case["read_len"]   # about 1.6 local alignments a mate in windows of 400 + L bases
        b, f = n * (32 + L + 60 + 1.6 * (400 + L) / 4 + 100), 12 * 1.6 * 1.5 * n * L * (400 + L)
    elif kind == "chains":
        n, L = case["n"], case["read_len"]   # one left and one right extension a chain, 13 operations a cell
        b, f = n * (24 + L + 4 * 24 + 2 * (L + 100) / 4 + 2 * 56), 13 * 0.75 * n * 2 * L * L / 12
    elif kind == "seed":
        n, L = case["n"], case["read_len"]   # about 5 backward extensions a base, 2 sectors and 40 operations each
        b, f = n * (L + 12 + 12 + 8 * 24) + 5 * n * L * 64, 40 * 5 * n * L
    else:
        b = f = 0.0
        for n in _request_sizes(case):
            for q in (100, 150, 250):
                x, y = _ext_work(n / 3, q, q * q, q + 55)
                b, f = b + x, f + y
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    return None
