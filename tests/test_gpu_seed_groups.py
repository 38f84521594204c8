"""The group-per-read SMEM kernel (eight threads a read) where it can go wrong,
against the oracle's restatement of SMEMFinder.findAllSMEMs: tandem repeats
with more candidates than one round (8) and than the shared-memory entries
(32) hold, reads shorter than a group, counts around a block's groups, a
sentinel in the middle of a block, and an index that the 32-byte blocks cannot
hold (a position in no bitstring), which keeps the 64-byte checkpoints."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(oracle_mod, n, seed):
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, 4, n).astype(np.uint8)
    for k in range(12):                      # tandem blocks, nested in length
        unit = rng.integers(0, 4, 2 + k % 5).astype(np.uint8)
        at = int(rng.integers(0, n - 2100))
        codes[at:at + 150 * (k + 2)] = np.resize(unit, 150 * (k + 2))
    return codes, oracle_mod.bwt_build(codes)


def _reads(codes, seed, n, lmax):
    rng = np.random.default_rng(seed)
    chunks, lens = [], []
    for r in range(n):
        L = int(rng.integers(0, 12)) if r % 9 == 0 else int(rng.integers(20, lmax))
        p = int(rng.integers(0, len(codes) - L))
        x = codes[p:p + L].copy()
        x[rng.random(L) < 0.01] = rng.integers(0, 4)
        x[rng.random(L) < 0.004] = 4
        chunks.append(x if r % 2 else np.where(x[::-1] < 4, 3 - x[::-1], 4).astype(np.uint8))
        lens.append(L)
    lens = np.array(lens, np.int32)
    off = np.concatenate([[0], np.cumsum(lens.astype(np.uint64))[:-1]]).astype(np.uint64)
    return np.concatenate(chunks + [np.zeros(1, np.uint8)]), off, lens


@pytest.mark.parametrize("wide", [False, True], ids=["blocks32", "checkpoints64"])
@pytest.mark.parametrize("n,lmax", [(1, 200), (15, 200), (17, 900), (2500, 260)])
def test_groups_equal_oracle(oracle_mod, wide, n, lmax):
    from swiftbwa_b200.alignment import Engine
    codes, idx = _index(oracle_mod, 40_000, 3)
    cp = np.concatenate([idx.cp, np.zeros(1, idx.cp.dtype)])     # one block past the end, holding the totals
    cp[-1]["counts"] = idx.cp[-1]["counts"] + [bin(int(b)).count("1") for b in idx.cp[-1]["bits"]]
    if wide:
        blk = len(idx.cp) // 3
        c = int(np.nonzero(cp[blk]["bits"])[0][0])
        b = int(cp[blk]["bits"][c])
        cp[blk]["bits"][c] = b & (b - 1)                         # one position in no bitstring
    ref = type(idx)(cp, idx.count, idx.length, idx.sentinel)
    bases, off, lens = _reads(codes, 100 + n, n, lmax)
    cap = 512
    exp, en, over = oracle_mod.smem_batch(ref, bases, off, lens, 15, cap=cap, n_threads=8, split_len=28, split_width=10)
    assert over == 0
    eng = Engine(0)
    try:
        eng.upload_bwt(cp, idx.count, idx.length, idx.sentinel)
        eng.profile(True)
        got, gn, goff = eng.smem_batch(bases, off, lens, 15, cap_per_read=cap, split_len=28)
        ran = [k for k in eng.profile_read() if k.startswith("smem_search")]
    finally:
        eng.close()
    assert ran == (["smem_search_cp64"] if wide else ["smem_search"])
    assert np.array_equal(gn, en)
    for r in range(n):
        assert np.array_equal(got[goff[r]:goff[r] + gn[r]], exp[r * cap:r * cap + en[r]]), f"read {r}"


def test_refused_upload_keeps_the_index(oracle_mod):
    """An index that the memory budget does not hold is refused before anything
    is freed: the one uploaded before it still gives its SMEMs."""
    from swiftbwa_b200 import abi
    from swiftbwa_b200.alignment import Engine, SWBError
    codes, idx = _index(oracle_mod, 40_000, 5)
    bases, off, lens = _reads(codes, 7, 40, 200)
    exp, en, _ = oracle_mod.smem_batch(idx, bases, off, lens, 15, cap=512, n_threads=8, split_len=28, split_width=10)
    budget = 24 << 20
    n_cp = budget * 5 // 4 // 64               # 1.25 budgets as checkpoints, 0.63 as 32-byte blocks
    big = np.zeros(n_cp, idx.cp.dtype)
    length = (n_cp - 1) * 64
    eng = Engine(0, mem_budget_bytes=budget)
    try:
        eng.upload_bwt(idx.cp, idx.count, idx.length, idx.sentinel)
        for _ in range(2):
            with pytest.raises(SWBError) as ei:
                eng.upload_bwt(big, np.array([0, 1, 2, 3, length]), length, 5)
            assert ei.value.status == abi.SWB_ERR_OOM
            got, gn, goff = eng.smem_batch(bases, off, lens, 15, cap_per_read=512, split_len=28)
            assert np.array_equal(gn, en)
            for r in range(len(lens)):
                assert np.array_equal(got[goff[r]:goff[r] + gn[r]], exp[r * 512:r * 512 + en[r]]), f"read {r}"
    finally:
        eng.close()
