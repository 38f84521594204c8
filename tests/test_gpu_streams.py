"""Calls of one context on several streams, and of several contexts on several
threads.  One context: a device entry returns while its pass runs, and the
calls after it, on other streams or through host entries, use the same
workspace.  Every call has to give the oracle's results.  Batches small enough
for a warp per task and large enough for the bins to leave rows out, each next
one larger (the workspace moves); the plain form; host batches of extensions
and of global alignments in between."""
import numpy as np
import pytest

import gen
from swiftbwa_b200.abi import EXT_RESULT_DTYPE, Scoring
from test_gpu_ext_skip import _tasks

pytestmark = pytest.mark.gpu


def test_calls_on_several_streams(oracle_mod):
    import torch
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default()
    eng = Engine(0)
    try:
        sets = []
        for k, (n, rep, qmax) in enumerate([(6000, 17, 250), (5000, 21, 140), (3000, 1, 300), (6000, 30, 200)]):
            bases, tasks = _tasks(3000 + k, n, qmax)
            exp, _ = oracle_mod.ext_batch(sc, bases, tasks, n_threads=8)
            t = np.tile(tasks, rep)
            sets.append((bases, t, np.tile(exp, rep), torch.from_numpy(bases).cuda(),
                         torch.from_numpy(t.view(np.uint8)).cuda()))
        streams = [torch.cuda.Stream() for _ in range(3)]
        torch.cuda.synchronize()
        runs = []
        for turn in range(8):
            bases, t, want, d_b, d_t = sets[turn % len(sets)]
            out = torch.full((len(t) * EXT_RESULT_DTYPE.itemsize,), 0x5A, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()             # (the fill ran on torch's stream; the passes need not be done)
            entry = eng.ext_batch_plain_device if turn == 5 else eng.ext_batch_device
            for _ in range(2):
                entry(sc, d_b.data_ptr(), d_t.data_ptr(), len(t), out.data_ptr(), streams[turn % 3].cuda_stream)
            runs.append((turn, out, want))
            if turn in (2, 6):
                b, tt, w = sets[1][0], sets[1][1][:20_000], sets[1][2][:20_000]
                assert np.array_equal(eng.ext_batch(sc, b, tt), w), f"host batch after turn {turn}"
                g = gen.global_tasks(7, 300)
                res, _ = eng.global_batch(sc, g["bases"], g["tasks"])
                eres, _, _ = oracle_mod.global_batch(sc, g["bases"], g["tasks"], n_threads=8)
                assert np.array_equal(res["score"], eres["score"])
        torch.cuda.synchronize()
        for turn, out, want in runs:
            got = out.cpu().numpy().view(EXT_RESULT_DTYPE)
            bad = np.nonzero(got != want)[0]
            assert bad.size == 0, f"turn {turn}: {bad.size} mismatches"
    finally:
        eng.close()


def test_passes_overlap_without_waiting_in_between(oracle_mod):
    """Four batches queued on four streams before any is waited for."""
    import torch
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default()
    bases, tasks = _tasks(3100, 6000, 250)
    exp, _ = oracle_mod.ext_batch(sc, bases, tasks, n_threads=8)
    eng = Engine(0)
    try:
        d_b = torch.from_numpy(bases).cuda()
        order = [np.random.default_rng(k).permutation(len(tasks) * 20) % len(tasks) for k in range(4)]
        ts = [torch.from_numpy(tasks[o].view(np.uint8)).cuda() for o in order]
        outs = [torch.zeros(len(o) * EXT_RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda") for o in order]
        streams = [torch.cuda.Stream() for _ in range(4)]
        torch.cuda.synchronize()
        for t, o, out, s in zip(ts, order, outs, streams):
            eng.ext_batch_device(sc, d_b.data_ptr(), t.data_ptr(), len(o), out.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        for o, out in zip(order, outs):
            assert np.array_equal(out.cpu().numpy().view(EXT_RESULT_DTYPE), exp[o])
    finally:
        eng.close()


def test_contexts_on_several_threads(oracle_mod):
    """Kernels whose shared memory a call sizes by its longest query, called from
    two threads with different lengths (each its own context)."""
    import threading
    from swiftbwa_b200.alignment import Engine
    sc = Scoring.default()
    work = []
    for k, qmax in enumerate((300, 3800)):
        e = gen.ext_tasks(40 + k, 40, qmax=qmax)
        g = gen.global_tasks(50 + k, 6000, qmax=40 if k else 250, retry=False)
        exp, _ = oracle_mod.ext_batch(sc, e["bases"], e["tasks"], n_threads=8)
        eres, _, _ = oracle_mod.global_batch(sc, g["bases"], g["tasks"], n_threads=8)
        work.append((e, exp, g, eres))
    errors = []

    def loop(e, exp, g, eres):
        eng = Engine(0)
        try:
            for turn in range(150):
                if not np.array_equal(eng.ext_batch(sc, e["bases"], e["tasks"]), exp):
                    raise AssertionError("extensions differ")
                if turn % 5 == 0 and not np.array_equal(eng.global_batch(sc, g["bases"], g["tasks"])[0]["score"],
                                                        eres["score"]):
                    raise AssertionError("global alignments differ")
        except Exception as x:   # noqa: BLE001 -- reported below, in the test's thread
            errors.append(x)
        finally:
            eng.close()

    th = [threading.Thread(target=loop, args=w) for w in work for _ in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors[0]
