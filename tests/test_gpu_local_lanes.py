"""The packed striped local SW kernels (8 threads play the reference's 16 SIMD
lanes) at the sizes where they can go wrong, against the oracle (the C++
restatement of LocalSWAligner.align): every stripe-count edge, targets around
the 8-column load blocks, fewer tasks than a warp holds, exact hits and hits
with one insertion (where the reverse pass may or may not stop early), and
scorings whose H + profile byte wraps."""
import numpy as np
import pytest

from swiftbwa_b200.abi import LOCAL_TASK_DTYPE, Scoring

pytestmark = pytest.mark.gpu

SCORINGS = [dict(), dict(a=2, b=8, o_ins=3, e_ins=2), dict(a=1, b=9), dict(a=1, b=1, o_ins=1, e_ins=1), dict(a=0)]


def _tasks(seed, qlens, tlens):
    rng = np.random.default_rng(seed)
    chunks, rows, off = [], [], 0
    for qlen in qlens:
        for k, tlen in enumerate(tlens):
            q = rng.integers(0, 4, qlen).astype(np.uint8)
            t = rng.integers(0, 4, tlen).astype(np.uint8)
            hit = q.copy()
            if k % 4 == 1 and qlen > 4:      # one base of the query missing from the target: an insertion
                hit = np.delete(hit, int(rng.integers(1, qlen - 1)))
            elif k % 4 == 2 and qlen > 4:    # one substitution
                hit[int(rng.integers(0, qlen))] ^= 1
            elif k % 4 == 3:                 # tandem repeat: many equal maxima
                q = np.resize(rng.integers(0, 4, 3).astype(np.uint8), qlen)
                hit = q
            at = int(rng.integers(0, max(tlen - len(hit), 0) + 1))
            n = min(len(hit), tlen - at)
            t[at:at + n] = hit[:n]
            chunks += [q, t]
            rows.append((off, off + qlen, qlen, tlen, int(rng.choice([0, 1, 10, 19])), 0))
            off += qlen + tlen
    return np.concatenate(chunks), np.array(rows, dtype=LOCAL_TASK_DTYPE)


@pytest.mark.parametrize("scoring", SCORINGS, ids=lambda s: "-".join(f"{k}{v}" for k, v in s.items()) or "default")
@pytest.mark.parametrize("n", [1, 3, None])
def test_stripe_and_block_edges(oracle_mod, scoring, n):
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default(**scoring)
    qlens = sorted({q for s in range(1, 17) for q in (16 * s - 15, 16 * s - 1, 16 * s)} | {250, 251, 257, 300})
    bases, tasks = _tasks(17, qlens, [1, 7, 8, 9, 16, 17, 40, 301])
    if n is not None:
        tasks = tasks[100:100 + n]
    eng = Engine(0)
    try:
        got = eng.local_batch(sc, bases, tasks)
        cells = eng.last_batch_stats()[1]
    finally:
        eng.close()
    exp, exp_cells = oracle_mod.local_batch(sc, bases, tasks, n_threads=8)
    bad = np.nonzero(got != exp)[0]
    assert bad.size == 0, f"{bad.size} mismatches, first {tasks[bad[:3]]}: {got[bad[:3]]} vs {exp[bad[:3]]}"
    assert cells == exp_cells
