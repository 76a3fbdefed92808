"""The resident loop's wait of a strip on its neighbour gives up with an error status (GPU test).

The self-test waits, through the loop's own wait, on words that nothing writes: the flag reads 1 after
the limit, the second wait ends at once because the flag is up, and the context still runs a solve.
"""
import time

import pytest
import torch

import adfwi_gb300 as A
from adfwi_gb300 import _native as N
from _cases import acoustic_problem

pytestmark = pytest.mark.gpu


def test_rows_that_nothing_writes_time_out_with_status():
    flag = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    row = torch.full((8,), 5.0, device="cuda:0")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    N.row_wait_selftest(200_000_000, flag, row)  # 0.2 s
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    assert int(flag.item()) == 1
    assert row.tolist() == [0.0] * 8  # both waits marked their block, and left the words' values
    assert 0.15 <= dt < 0.39, dt  # one limit, not two
    model, survey, prop = acoustic_problem(A, ns=2, nt=60, seed=3)
    rec = prop.forward()
    assert torch.isfinite(rec["p"]).all()


def test_row_wait_selftest_rejects_bad_arguments():
    flag = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    row = torch.zeros(8, device="cuda:0")
    for limit in (0, 3_000_000_000):
        with pytest.raises(RuntimeError):
            N.row_wait_selftest(limit, flag, row)
