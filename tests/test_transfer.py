"""The team of copy threads (csrc/transfer.cu) on a stand-in of the CUDA runtime, compiled for the host.

* Uploads from several pieces and downloads arrive, below and above the size from which the team copies.
* Threads that can make no stream or pin no blocks leave their share to the others; when none can, the
  runtime's own copy does the work, and no error of the attempt stays behind.
* An error of a copy itself is reported.
"""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from nanoshaper_b200 import build

ROOT = Path(__file__).resolve().parents[1]
MANY = 1 << 20


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = tmp_path_factory.mktemp("transfer") / "transfer.so"
    cuda = Path(build._nvcc()).resolve().parents[1]
    # -Bsymbolic: the stand-in's calls, also where another library has loaded the real runtime
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I", str(build.CSRC), "-I",
                    str(cuda / "include"), str(ROOT / "tests" / "cxx" / "transfer_check.cpp"), "-o", str(out)], check=True)
    fn = ctypes.CDLL(str(out)).transfer_check
    fn.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    fn.restype = None

    def run(n_bytes, to_device, allocs=MANY, streams=MANY, failing_copy=0):
        got = np.zeros(4, np.int64)
        fn(n_bytes, int(to_device), allocs, streams, failing_copy, got.ctypes.data)
        return got.tolist()

    return run


@pytest.mark.parametrize("to_device", [False, True])
@pytest.mark.parametrize("n_bytes", [1 << 10, (1 << 20) - 1001, 1 << 20, (1 << 20) + 7, (37 << 20) + 12345])
def test_copies_arrive(n_bytes, to_device, check):
    rc, differ, last, pageable = check(n_bytes, to_device)
    assert (rc, differ, last) == (0, 0, 0)
    assert (pageable == 0) == (n_bytes + 1000 >= 1 << 20)


@pytest.mark.parametrize("to_device", [False, True])
@pytest.mark.parametrize("allocs,streams", [(0, MANY), (1, MANY), (2, MANY), (3, MANY), (7, MANY), (MANY, 0), (MANY, 1)])
def test_threads_that_cannot_start(allocs, streams, to_device, check):
    for _ in range(20):  # which thread gets the blocks differs
        rc, differ, last, pageable = check((5 << 20) + 3, to_device, allocs, streams)
        assert (rc, differ, last) == (0, 0, 0)
        if min(allocs // 2, streams) == 0:
            assert pageable == (4 if to_device else 2)  # three pieces and the small copy


@pytest.mark.parametrize("to_device", [False, True])
def test_a_failing_copy_is_reported(to_device, check):
    assert check(5 << 20, to_device, failing_copy=3)[0] == 999  # cudaErrorUnknown
