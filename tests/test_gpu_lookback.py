"""The look-back offsets of the one-pass kernels (csrc/kernels/lookback.cuh) by themselves.

* Whether a block goes on is its thread 0's decision, whatever the other threads would read: the error
  word may change while a block reads it, and a block must not part before a warp-wide exchange.  One
  that does not go on leaves a count of 0 for its ticket.
* A wait for a ticket that nothing publishes runs out: the blocks return -1, set the error word, and the
  kernel ends.
"""
import ctypes
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
THREADS = 256


@pytest.fixture(scope="module")
def lookback(tmp_path_factory):
    from nanoshaper_b200 import build
    out = tmp_path_factory.mktemp("lookback") / "lookback.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-I", str(build.CSRC),
                    str(ROOT / "tests" / "cxx" / "lookback_check.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("err0,cond0,goes_on", [(0, 1, True), (8, 1, False), (0, 0, False)])
def test_thread_0_decides(err0, cond0, goes_on, lookback):
    import torch
    err = torch.full((THREADS,), 8 - err0, dtype=torch.int32, device="cuda")
    cond = torch.full((THREADS,), 1 - cond0, dtype=torch.int32, device="cuda")
    err[0], cond[0] = err0, cond0
    out = torch.full((THREADS,), -1, dtype=torch.int32, device="cuda")
    state = torch.zeros(4, dtype=torch.int64, device="cuda")
    ticket = torch.full((1,), 2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lookback.decide(_ptr(state), _ptr(ticket), _ptr(err), _ptr(cond), _ptr(out)) == 0
    assert (out == (3 if goes_on else 0)).all() and ticket.item() == 3
    assert state.tolist() == [0, 0, 0 if goes_on else 1 << 62, 0]


@pytest.mark.parametrize("first", [0, 3])
def test_wait_for_a_missing_ticket_runs_out(first, lookback):
    """Three blocks with the tickets from `first` on: with 0 all of them are there; with 3, tickets 0 to 2
    are never taken."""
    import torch
    words = 8
    state = torch.zeros(words, dtype=torch.int64, device="cuda")
    ticket = torch.full((1,), first, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((words,), -7, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert lookback.offsets(_ptr(state), _ptr(ticket), _ptr(err), words, 3, _ptr(out)) == 0
    got = out.tolist()
    if first == 0:
        per_ticket = THREADS // 32  # one item per warp
        assert got == [0, per_ticket, 2 * per_ticket] + [-7] * 5 and err.item() == 0
    else:
        assert got == [-7] * 3 + [-1] * 3 + [-7] * 2 and err.item() == 8
