"""Contexts on a caller's stream.

* On the default stream (0), whose work nothing else waits for: a context that is destroyed, or moved
  to another stream, right after calls that leave work behind (an upload from pinned memory, cavity
  filling) hands its memory on only when that work is done, so that contexts made at once get their
  own results.
* Cavity detection returns when nothing of it is left on the stream.
"""
import ctypes

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

pytestmark = pytest.mark.gpu

FLAGS = 1 | 2 | 4  # status map, triangulation rays, epsilon maps


def _surface(n_atoms, seed, scale):
    nb.reset_seed()
    cf = nb.ConfigFile(text="Surface = ses\nProbe_Radius = 1.4\nAccurate_Triangulation = true\nTriangulation = true\n")
    surf = nb.surfaceFactory().create(cf, nb.DelPhiShared(generator.rsa_globule(n_atoms, seed), scale, 80.0))
    surf.build()
    return surf


class _Ctx:
    """A context on the default stream, holding the patch set of a surface in pinned memory."""

    def __init__(self, surf, pinned, stream=0):
        L = self.L = N.lib()
        self.surf = surf
        self.h = ctypes.c_void_p()
        N.check(L.nsg_ctx_create(0, ctypes.byref(self.h)), "create")
        N.check(L.nsg_set_stream(self.h, ctypes.c_void_p(stream)), "stream")
        N.check(L.nsg_set_grid(self.h, ctypes.byref(surf.delphi.grid)), "grid")
        p = surf.patches
        f64, i32, pool, flag = (t.data_ptr() for t in pinned)
        N.check(L.nsg_upload_patches(self.h, p.n, f64, i32, len(p.pool), pool, flag, p.probe), "upload")

    def cast(self):
        vol, ncav = ctypes.c_double(), ctypes.c_int()
        N.check(self.L.nsg_raycast(self.h, FLAGS, 0, ctypes.byref(vol)), "raycast")
        N.check(self.L.nsg_cavities(self.h, 40.0, ctypes.byref(ncav)), "cavities")
        return vol.value, ncav.value

    def bits(self):
        g = self.surf.delphi.grid
        w = np.empty((g.nx + 31) // 32 * g.ny * g.nz, np.uint32)
        N.check(self.L.nsg_download_insideness(self.h, N.ptr(w)), "bits")
        return w

    def close(self):
        N.check(self.L.nsg_ctx_destroy(self.h), "destroy")


@pytest.fixture(scope="module")
def case(native_lib):
    import torch
    surf = _surface(4000, 3, 3.0)
    p = surf.patches
    pinned = [torch.from_numpy(a).pin_memory() for a in (p.f64, p.i32, p.pool, p.pool_flag)]
    ctx = _Ctx(surf, pinned)
    want = ctx.cast() + (ctx.bits(),)
    ctx.close()
    return surf, pinned, want


def _same(ctx, want):
    assert ctx.cast() == want[:2]
    assert np.array_equal(ctx.bits(), want[2])


def test_destroyed_on_the_default_stream(case):
    surf, pinned, want = case
    for _ in range(3):
        left = _Ctx(surf, pinned)  # its upload may still be on the way
        left.close()
        ctx = _Ctx(surf, pinned)
        ctx.cast()                 # leaves the filling of the bits behind
        ctx.close()
        last = _Ctx(surf, pinned)
        _same(last, want)
        last.close()


def test_moved_between_streams(case):
    import torch
    surf, pinned, want = case
    other = torch.cuda.Stream()
    ctx = _Ctx(surf, pinned)
    N.check(ctx.L.nsg_set_stream(ctx.h, ctypes.c_void_p(other.cuda_stream)), "stream")
    _same(ctx, want)
    N.check(ctx.L.nsg_set_stream(ctx.h, None), "stream")
    _same(ctx, want)
    ctx.close()


def test_cavity_detection_leaves_nothing_on_the_stream(native_lib):
    import torch
    surf = _surface(20000, 1, 4.0)
    p = surf.patches
    pinned = [torch.from_numpy(a).pin_memory() for a in (p.f64, p.i32, p.pool, p.pool_flag)]
    stream = torch.cuda.Stream()
    ctx = _Ctx(surf, pinned, stream.cuda_stream)
    for _ in range(3):
        ctx.cast()
        assert stream.query()
    ctx.close()
