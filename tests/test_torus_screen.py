"""The single-precision screen of torus candidates (csrc/torus_screen.h) on the CPU, against the
double-precision path compiled for the host: a candidate with a feasible hit is never dropped, on
every panel, for on-node and shifted rays, at molecular size (dense and loose globules, small and
large probes, far from the origin) and at a tenth and ten times of it, where the solver's absolute
thresholds make its roots inexact and the screen leaves its distance test out; at molecular size it
keeps a fifth of the candidates of a dense globule."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = tmp_path_factory.mktemp("screen") / "screen.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    str(ROOT / "nanoshaper_b200" / "csrc"), str(ROOT / "tests" / "cxx" / "torus_screen_check.cpp"),
                    "-o", str(out)], check=True)
    fn = ctypes.CDLL(str(out)).torus_screen_check
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                   ctypes.c_double, ctypes.c_int, ctypes.c_double, ctypes.c_void_p]
    fn.restype = None
    return fn


@pytest.mark.parametrize("n,probe,scale,inflate,unit,shift", [
    (2, 1.4, 6.0, 1.37, 1.0, 0.0), (60, 1.4, 3.0, 1.37, 1.0, 0.0), (400, 1.4, 2.0, 1.37, 1.0, 700.0),
    (300, 0.7, 3.0, 1.6, 1.0, 0.0), (300, 3.0, 2.5, 1.37, 1.0, 0.0), (300, 5.0, 2.0, 1.37, 1.0, 0.0),
    (150, 1.4, 3.0, 2.2, 1.0, -300.0), (200, 1.4, 2.5, 1.37, 0.1, 0.0), (200, 1.4, 2.5, 1.37, 10.0, 0.0),
    (100, 5.0, 2.5, 1.6, 10.0, 0.0)])
def test_screen_keeps_every_hit(n, probe, scale, inflate, unit, shift, check):
    if n == 2:
        atoms = np.array([[0.0, 0.0, 0.0, 1.7], [2.1, 0.4, -0.3, 1.5]])  # one full torus
    else:
        atoms = generator.rsa_globule(n, n + int(10 * probe), inflate=inflate)
    atoms[:, :3] += shift
    atoms = atoms * unit
    ds = nb.DelPhiShared(atoms, scale / unit, 80.0)
    seed = ctypes.c_int64(1234)
    N.check(N.lib().nsg_jitter_atoms(N.ptr(ds.atoms), len(ds.atoms), 1e-4, ctypes.byref(seed)), "jitter")
    p = nb.build_ses_patches(ds.atoms, probe * unit, 1)
    counts = np.zeros(4, np.int64)
    for panel in range(3):
        for delta in (0.0, 1e-10 - ds.grid.hside):
            check(ctypes.addressof(ds.grid), p.n, N.ptr(p.f64), N.ptr(p.i32), N.ptr(p.pool), N.ptr(p.pool_flag),
                  probe * unit, panel, delta, N.ptr(counts))
    candidates, with_hit, kept, lost = counts.tolist()
    assert with_hit > 0 and lost == 0
    assert with_hit <= kept <= candidates
    if unit == 1.0 and inflate == 1.37 and probe == 1.4 and n > 2:
        assert kept < 0.3 * candidates
