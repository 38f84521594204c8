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
            got[budget] = gen.ext_batch_binned(eng, sc, wl.bases, wl.tasks)
        except SWBError as e:
            got[budget] = e.status
        finally:
            eng.close()
    assert np.array_equal(got[25 * n], got[0])
    assert isinstance(got[23 * n], int) and got[23 * n] == abi.SWB_ERR_OOM
