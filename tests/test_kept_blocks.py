"""Kept memory blocks (csrc/kept_blocks.h): a request takes the smallest block that is large enough, and
what is kept stays within its bound."""
import ctypes
import subprocess
from pathlib import Path

from nanoshaper_b200 import build

ROOT = Path(__file__).resolve().parents[1]


def test_smallest_block_and_bound(tmp_path):
    out = tmp_path / "kept.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(build.CSRC),
                    str(ROOT / "tests" / "cxx" / "kept_blocks_check.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    for name in ("give", "take", "bytes"):
        getattr(lib, name).restype = ctypes.c_long
        getattr(lib, name).argtypes = [ctypes.c_long] * {"give": 3, "take": 1, "bytes": 0}[name]
    most = 1000
    assert lib.take(1) == 0
    assert lib.give(1, 600, most) and lib.give(2, 100, most) and lib.give(3, 300, most)
    assert not lib.give(4, 1, most) and lib.bytes() == 1000
    assert lib.take(50) == 2       # not the first that is large enough
    assert lib.take(301) == 1
    assert lib.take(301) == 0
    assert lib.give(5, 300, most)  # equal sizes: either
    assert {lib.take(300), lib.take(300)} == {3, 5}
    assert lib.bytes() == 0
