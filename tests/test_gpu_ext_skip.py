"""Extension rows left out (those before the first mismatch, and those after
which nothing can change) against the oracle, on tasks that reach the rules'
edges: exact matches, a first mismatch or N at every position, an indel right
at the start or the end, two close mismatches, tandem repeats, targets shorter
than the query, bands from one column up, h0 from 1, queries kept as rings, and
scorings with free gap opening, expensive mismatches or a match score above the
gap costs.  With profiling on every row is computed and the cell count is the
oracle's; without, the results must be the same.  Batches of three sizes: one
that runs a warp per extension, one that runs the length bins with every first
row, and one (the tasks repeated) large enough for the bins to leave them out."""
import numpy as np
import pytest

import gen
from swiftbwa_b200.abi import (EXT_TASK_DTYPE, SWB_Q_REVERSE, SWB_T_COMPLEMENT, SWB_T_FROM_REF, SWB_T_REVERSE,
                               Scoring)

pytestmark = pytest.mark.gpu

SCORINGS = [dict(), dict(o_ins=0, o_del=0), dict(a=3, b=2, o_ins=2, e_ins=1, o_del=1, e_del=1), dict(b=60, zdrop=20),
            dict(a=1, b=0, o_ins=1, o_del=3), dict(a=2, b=9, o_ins=5, e_ins=3, o_del=2, e_del=4, zdrop=0)]


def _tasks(seed, n, qmax):
    rng = np.random.default_rng(seed)
    chunks, rows, off = [], [], 0
    for k in range(n):
        qlen = int(rng.integers(1, 6)) if k % 17 == 0 else int(rng.integers(6, qmax + 1))
        q = (gen.tandem(rng, qlen) if k % 5 == 0 else rng.integers(0, 4, qlen)).astype(np.uint8)
        kind = k % 8
        t = q.copy()
        at = int(rng.integers(0, qlen))
        if kind == 1:
            t[at] = (t[at] + 1) & 3
        elif kind == 2:
            q[at] = 4
        elif kind == 3:
            t = np.insert(t, at, rng.integers(0, 4, int(rng.integers(1, 4)))).astype(np.uint8)
        elif kind == 4:
            t = np.delete(t, slice(at, at + int(rng.integers(1, 4))))
        elif kind == 5:
            t[at] = (t[at] + 1) & 3
            a2 = min(qlen - 1, at + int(rng.integers(1, 5)))
            t[a2] = (t[a2] + 2) & 3
        elif kind == 6:
            t[rng.random(qlen) < 0.03] = rng.integers(0, 4)
        w = int(rng.choice([1, 2, 3, 7, 20, 100]))
        tail = int(rng.integers(0, w + 1)) if k % 3 else w
        t = np.concatenate([t, gen.tandem(rng, tail) if k % 4 == 0 else rng.integers(0, 4, tail)]).astype(np.uint8)
        if k % 11 == 0:
            t = t[:int(rng.integers(0, qlen + 1))]
        flags = 0
        if rng.random() < 0.3:
            q, flags = q[::-1].copy(), flags | SWB_Q_REVERSE
        if rng.random() < 0.3:
            t, flags = t[::-1].copy(), flags | SWB_T_REVERSE
        if rng.random() < 0.2:
            t, flags = np.where(t < 4, 3 - t, 4).astype(np.uint8), flags | SWB_T_COMPLEMENT
        chunks += [q, t]
        rows.append((off, off + len(q), len(q), len(t), w, int(rng.choice([1, 2, 8, 19, 60, 150])),
                     int(rng.integers(0, 11)), flags))
        off += len(q) + len(t)
    return np.concatenate(chunks + [np.zeros(1, np.uint8)]), np.array(rows, dtype=EXT_TASK_DTYPE)


@pytest.mark.parametrize("bins", [None, [24, 100, 232]], ids=["default", "coarse"])
@pytest.mark.parametrize("si", range(len(SCORINGS)))
@pytest.mark.parametrize("qmax", [140, 700])
def test_rows_left_out(oracle_mod, si, qmax, bins):
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default(**SCORINGS[si])
    bases, tasks = _tasks(900 + 10 * si + qmax, 6000, qmax)
    exp, cells = oracle_mod.ext_batch(sc, bases, tasks, n_threads=8)
    eng = Engine(0)

    def check(got, want, t):
        bad = np.nonzero(got != want)[0]
        assert bad.size == 0, f"{len(t)}: {bad.size} mismatches, first {t[bad[:3]]}: {got[bad[:3]]} vs {want[bad[:3]]}"

    try:
        if bins:
            eng.set_ext_bins(bins)
        for n, rep in ((1500, 1), (6000, 1), (6000, 17)):
            t, want = np.tile(tasks[:n], rep), np.tile(exp[:n], rep)
            check(gen.ext_batch_device(eng, sc, bases, t), want, t)
            eng.profile(True)
            eng.profile_reset()
            every = gen.ext_batch_device(eng, sc, bases, t)
            prof = eng.profile_read()
            eng.profile(False)
            check(every, want, t)
            if n == 6000:
                assert sum(v[2] for k, v in prof.items() if k.startswith("ext_")) == cells * rep
            check(eng.ext_batch(sc, bases, t), want, t)
            if n == 6000:
                assert eng.last_batch_stats()[1] == cells * rep
    finally:
        eng.close()


def _on_reference(rng, bases, tasks):
    """The tasks with their targets on a resident strand where they hold no N
    (each behind 0-15 bases, so that spans begin anywhere in a word)."""
    t, parts, at = tasks.copy(), [], 0
    for k, x in enumerate(tasks):
        span = bases[int(x["t_off"]):int(x["t_off"]) + int(x["tlen"])]
        if x["tlen"] == 0 or (span > 3).any():
            continue
        gap = int(rng.integers(0, 16))
        parts += [rng.integers(0, 4, gap).astype(np.uint8), span]
        t["t_off"][k] = at + gap
        t["flags"][k] |= SWB_T_FROM_REF
        at += gap + len(span)
    ref = np.concatenate(parts)
    return t, gen.pack_ref(ref), len(ref)


@pytest.mark.parametrize("si", [0, 2, 3])
def test_rows_left_out_on_the_reference(oracle_mod, si):
    """The same rules where targets are spans of the packed reference, either
    strand and direction, in a pass that leaves rows out in the bins and in one
    with a warp per task."""
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default(**SCORINGS[si])
    bases, tasks = _tasks(1700 + si, 6000, 250)
    tasks, pac, ref_bases = _on_reference(np.random.default_rng(si), bases, tasks)
    assert ((tasks["flags"] & SWB_T_FROM_REF) != 0).sum() > 4000
    exp, _ = oracle_mod.ext_batch(sc, bases, tasks, pac=pac, ref_bases=ref_bases, n_threads=8)
    eng = Engine(0)
    try:
        eng.upload_reference(pac, ref_bases)
        for n, rep in ((3000, 1), (6000, 17)):
            t, want = np.tile(tasks[:n], rep), np.tile(exp[:n], rep)
            got = gen.ext_batch_device(eng, sc, bases, t)
            bad = np.nonzero(got != want)[0]
            assert bad.size == 0, f"{len(t)}: {bad.size} mismatches, first {t[bad[:3]]}: {got[bad[:3]]} vs {want[bad[:3]]}"
    finally:
        eng.close()


def test_chains_and_server_report_every_row(oracle_mod):
    """More tasks than the warp-per-task passes take: the cells that the chains
    and the request loop report are the oracle's."""
    from swiftbwa_b200 import workloads as W
    from swiftbwa_b200.alignment import Engine
    from swiftbwa_b200.serving import Server
    sc = Scoring.default()
    eng = Engine(0)
    try:
        ref = W.reference(W.SEED_BASE + 53, 300_000, tandem_frac=0.05)
        wl = W.chains(ref, 91, 9000, 150, sub=0.03, indel=0.01, spurious_frac=0.3, a=sc.a)
        eng.upload_reference(ref.pac, ref.n)
        eng.extend_chains(sc, wl.bases, wl.seeds, wl.chains, ref.n)
        _, _, cells = oracle_mod.extend_batch(sc, wl.bases, ref.pac, ref.n, wl.seeds, wl.chains, n_threads=8)
        assert eng.last_batch_stats()[1] == cells
        bases, tasks = _tasks(977, 6000, 140)
        exp, cells = oracle_mod.ext_batch(sc, bases, tasks, n_threads=8)
        srv = Server(eng, sc)
        try:
            got, _, _ = srv.wait(srv.submit(bases, tasks))
            assert np.array_equal(got, exp)
            assert srv.stats()["cells"] == cells
        finally:
            srv.stop()
    finally:
        eng.close()
