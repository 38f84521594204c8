"""The band-doubling retry of CIGARGenerator.generate at the width where a wider
band still changes the matrix: w = qlen - 1 covers every row, but the first
row's initialisation ends one column short, so the next attempt may trace
another path.  Against the oracle, with free gap opening, where that column
can be on the best path."""
import numpy as np
import pytest

from swiftbwa_b200.abi import GLOBAL_TASK_DTYPE, SWB_GLB_RETRY, Scoring

pytestmark = pytest.mark.gpu


def test_retry_at_the_width_of_the_query(oracle_mod):
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default(o_ins=0, o_del=0)
    rng = np.random.default_rng(5)
    chunks, rows, off = [], [], 0
    for k in range(4000):
        q, t = int(rng.integers(2, 8)), int(rng.integers(1, 8))
        chunks.append(rng.integers(0, 4, q + t).astype(np.uint8))
        rows.append((off, off + q, q, t, max(q, t) - 1 - (k % 3 == 0), 100, SWB_GLB_RETRY, 0))
        off += q + t
    bases = np.concatenate(chunks)
    tasks = np.array([r for r in rows if r[4] >= 1], dtype=GLOBAL_TASK_DTYPE)
    eres, ecig, cells = oracle_mod.global_batch(sc, bases, tasks, n_threads=8)
    eng = Engine(0)
    try:
        res, cig = eng.global_batch(sc, bases, tasks)
        assert eng.last_batch_stats()[1] == cells
    finally:
        eng.close()
    for k in range(len(tasks)):
        o, n, eo, en = (int(x) for x in (res["cigar_off"][k], res["n_cigar"][k], eres["cigar_off"][k], eres["n_cigar"][k]))
        assert (int(res["score"][k]), n) == (int(eres["score"][k]), en), tasks[k]
        assert np.array_equal(cig[o:o + n], ecig[eo:eo + en]), tasks[k]
