"""One warp per alignment NW + traceback (small batches) against the oracle
(the C++ restatement of GlobalAligner.align and of CIGARGenerator.generate's
retry): query lengths at the edges of a lane's columns and of the kernel's
instances, targets around the 32-row load blocks, bands from one column to the
whole matrix with the start column inside and at the edge of a lane, retries,
one alignment alone, and scorings with free gap opening.  Repeated past the size
where one thread runs an alignment, the results must be the same."""
import numpy as np
import pytest

import gen
from swiftbwa_b200.abi import GLOBAL_TASK_DTYPE, SWB_GLB_RETRY, SWB_Q_REVERSE, SWB_T_COMPLEMENT, Scoring

pytestmark = pytest.mark.gpu

SCORINGS = [dict(), dict(o_ins=0, o_del=0), dict(a=2, b=3, o_ins=5, e_ins=2, o_del=4, e_del=3)]


def _tasks(seed, qmax):
    rng = np.random.default_rng(seed)
    qlens = [q for q in (1, 2, 4, 5, 6, 31, 32, 33, 63, 127, 128, 129, 150, 159, 160, 161, 191, 192, 193, 255, 256)
             if q <= qmax]
    chunks, rows, off = [], [], 0
    for q in qlens:
        for k in range(40):
            x = (gen.tandem(rng, q) if k % 6 == 0 else rng.integers(0, 4, q)).astype(np.uint8)
            t = gen.mutate(rng, x, sub=0.04, indel=float(rng.choice([0.0, 0.01, 0.05])))
            if k % 10 == 3:
                t = rng.integers(0, 4, int(rng.choice([1, 31, 32, 33, 64, 65]))).astype(np.uint8)
            if len(t) == 0:
                t = np.array([2], np.uint8)
            x[rng.random(q) < 0.02] = 4
            flags = (SWB_GLB_RETRY if k % 2 else 0) | (SWB_Q_REVERSE if k % 5 == 1 else 0) | \
                    (SWB_T_COMPLEMENT if k % 7 == 2 else 0)
            chunks += [x, t]
            rows.append((off, off + q, q, len(t), int(rng.choice([1, 2, 3, 4, 5, 8, 30, 100, 400])),
                         int(rng.integers(-10, q + 1)), flags, 0))
            off += q + len(t)
    return np.concatenate(chunks), np.array(rows, dtype=GLOBAL_TASK_DTYPE)


def _same(tag, tasks, got, exp, rep=1):
    res, cig = got
    eres, ecig = exp
    n = len(eres)
    for f in ("score", "n_cigar", "w_used", "attempts"):
        want = np.tile(eres[f], rep)
        bad = np.nonzero(res[f] != want)[0]
        assert bad.size == 0, f"{tag}: {f} differs for {bad.size}, first {tasks[bad[0]]}"
    for k in range(len(res)):
        o, c, eo = int(res["cigar_off"][k]), int(res["n_cigar"][k]), int(eres["cigar_off"][k % n])
        assert np.array_equal(cig[o:o + c], ecig[eo:eo + c]), f"{tag}: task {k}"


@pytest.mark.parametrize("si", range(len(SCORINGS)))
@pytest.mark.parametrize("qmax", [128, 160, 192, 256])
def test_warp_alignments_equal_oracle(oracle_mod, si, qmax):
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default(**SCORINGS[si])
    bases, tasks = _tasks(70 + si + qmax, qmax)
    eres, ecig, cells = oracle_mod.global_batch(sc, bases, tasks, n_threads=8)
    eng = Engine(0)
    try:
        _same("batch", tasks, eng.global_batch(sc, bases, tasks), (eres, ecig))
        assert eng.last_batch_stats()[1] == cells
        one = eng.global_batch(sc, bases, tasks[-3:-2])
        assert int(one[0]["score"][0]) == int(eres["score"][-3])
        if qmax == 160 and si == 0:
            rep = 131072 // len(tasks) + 2
            res, cig = eng.global_batch(sc, bases, np.tile(tasks, rep))
            for f in ("score", "n_cigar", "w_used", "attempts"):
                assert np.array_equal(res[f], np.tile(eres[f], rep)), f
            _same("threads", tasks, (res[:len(tasks)], cig), (eres, ecig))
    finally:
        eng.close()
