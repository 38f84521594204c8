"""Calls at the edge of a context's memory budget: what a pass takes on top of
the least it needs is given up before the call is refused."""
import numpy as np
import pytest

import gen
from swiftbwa_b200 import abi
from swiftbwa_b200.abi import Scoring

pytestmark = pytest.mark.gpu


def test_extension_pass_without_room_for_rows_left_out():
    """24 bytes a task are the keys, the order and the sort's copies of them; the
    26 with the rows left out do not fit the budget."""
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.alignment import Engine, SWBError
    n = 2_000_000
    ref = W.reference(W.SEED_BASE + 61, 2_000_000)
    wl = W.uneven(ref, 62, n, qmin=30, qmax=60, wmin=5, wmax=20)
    sc = Scoring.default()
    got = {}
    for budget in (0, 25 * n, 23 * n):
        eng = Engine(0, mem_budget_bytes=budget + (1 << 20 if budget else 0))
        try:
            eng.upload_reference(ref.pac, ref.n)
            got[budget] = gen.ext_batch_device(eng, sc, wl.bases, wl.tasks)
        except SWBError as e:
            got[budget] = e.status
        finally:
            eng.close()
    assert np.array_equal(got[25 * n], got[0])
    assert isinstance(got[23 * n], int) and got[23 * n] == abi.SWB_ERR_OOM


def _least_budget(call, lo, hi, step=1 << 16):
    """The smallest budget (to `step`) with which call(budget) is not refused."""
    while hi - lo > step:
        mid = (lo + hi) // 2
        if call(mid) is None:
            lo = mid
        else:
            hi = mid
    return hi


def test_rescue_without_room_for_the_packed_regions(oracle_mod):
    """A call whose mates find nothing needs everything but the packed copy of
    the regions: with the least budget for it, the mates that find regions get
    them too."""
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.alignment import Engine, SWBError
    ref = W.reference(W.SEED_BASE + 63, 500_000)
    wl = W.rescue_jobs(ref, 64, 12_000, 100, n_contigs=3)
    args = (wl.bases, wl.jobs, wl.templates, wl.mate_regions, wl.stats, wl.primary, wl.contig_offsets,
            wl.contig_lengths, wl.ref.n)
    sc, none = Scoring.default(), Scoring.default(min_seed_len=1000)

    def call(budget, scoring):
        eng = Engine(0, mem_budget_bytes=budget)
        try:
            eng.upload_reference(ref.pac, ref.n)
            return eng.mate_rescue(scoring, *args)
        except SWBError as e:
            assert e.status == abi.SWB_ERR_OOM
            return None
        finally:
            eng.close()

    least = _least_budget(lambda b: call(b, none), 1 << 20, 1 << 30)
    assert int(call(least, none)[1].sum()) == 0
    got = call(least, sc)
    assert got is not None, "refused for want of room for the packed regions"
    exp, en, _, _ = oracle_mod.mate_rescue_batch(sc, wl.bases, wl.ref.pac, wl.ref.n, wl.jobs, wl.templates,
                                                 wl.mate_regions, wl.stats, wl.primary, wl.contig_offsets,
                                                 wl.contig_lengths, n_threads=8)
    assert np.array_equal(got[1], en) and int(en.sum()) * abi.RESCUED_DTYPE.itemsize > 1 << 18
    for j, job in enumerate(wl.jobs):
        o, k = 4 * int(job["tmpl_off"]), int(en[j])
        assert np.array_equal(got[0][o:o + k], exp[o:o + k]), j


def test_global_batch_whose_warps_would_take_the_long_queries_scratch(oracle_mod):
    """3000 short alignments and a long one (64 slots of 4 MB): the short ones'
    backpointers take 15 MB with a warp each and 2 MB with a thread each, and the
    budget leaves 8 MB."""
    from swiftbwa_b200.alignment import Engine
    rng = np.random.default_rng(65)
    L = 2000
    rows = [(0, L, L, L, 50, 0, 0, 0)]
    q = rng.integers(0, 4, L).astype(np.uint8)
    t = q.copy()
    t[rng.random(L) < 0.03] = 2
    chunks, off = [q, t], 2 * L
    for _ in range(3000):
        x = rng.integers(0, 4, 32).astype(np.uint8)
        chunks += [x, gen.mutate(rng, np.resize(x, 40), sub=0.03, indel=0.0)]
        rows.append((off, off + 32, 32, len(chunks[-1]), 30, 0, 0, 0))
        off += 32 + len(chunks[-1])
    bases, tasks = np.concatenate(chunks), np.array(rows, dtype=abi.GLOBAL_TASK_DTYPE)
    sc = Scoring.default()
    eres, ecig, _ = oracle_mod.global_batch(sc, bases, tasks, n_threads=8)
    least = 64 * ((L + 1) * 8 + 2 * L + L * L)
    eng = Engine(0, mem_budget_bytes=2 * (least + (8 << 20)))
    try:
        res, cig = eng.global_batch(sc, bases, tasks)
    finally:
        eng.close()
    for f in ("score", "n_cigar", "w_used", "attempts"):
        assert np.array_equal(res[f], eres[f]), f
    for k in range(len(tasks)):
        o, n, eo = int(res["cigar_off"][k]), int(res["n_cigar"][k]), int(eres["cigar_off"][k])
        assert np.array_equal(cig[o:o + n], ecig[eo:eo + n]), k


def test_host_batch_without_room_for_rows_left_out(oracle_mod):
    """The pipelined host entry (several chunks, two orders) with the least budget
    that it is not refused."""
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.alignment import Engine, SWBError
    ref = W.reference(W.SEED_BASE + 67, 2_000_000)
    wl = W.uneven(ref, 68, 600_000, qmin=30, qmax=60, wmin=5, wmax=20)
    sc = Scoring.default()

    def call(budget):
        eng = Engine(0, mem_budget_bytes=budget)
        try:
            eng.upload_reference(ref.pac, ref.n)
            return eng.ext_batch(sc, wl.bases, wl.tasks), eng.last_batch_stats()[1]
        except SWBError as e:
            assert e.status == abi.SWB_ERR_OOM
            return None
        finally:
            eng.close()

    got, cells = call(_least_budget(call, 1 << 20, 1 << 28))
    exp, want = oracle_mod.ext_batch(sc, wl.bases, wl.tasks, pac=ref.pac, ref_bases=ref.n, n_threads=8)
    assert np.array_equal(got, exp) and cells == want
