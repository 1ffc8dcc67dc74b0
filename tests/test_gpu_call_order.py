"""Calls of one context in orders that a program may well make, although the Python classes do not.

* Patches uploaded or bound between a cast and its triangulation: the triangulation is that of the
  cast.
* A batch that is refused (more than 2^31 rays) leaves the grid before in force.
"""
import ctypes

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

pytestmark = pytest.mark.gpu


def _surface(n_atoms, seed, scale=2.0, perfil=80.0):
    nb.reset_seed()
    cf = nb.ConfigFile(text="Surface = ses\nProbe_Radius = 1.4\nAccurate_Triangulation = true\nTriangulation = true\n")
    surf = nb.surfaceFactory().create(cf, nb.DelPhiShared(generator.rsa_globule(n_atoms, seed), scale, perfil))
    surf.build()
    return surf


def _upload(handle, p):
    return N.lib().nsg_upload_patches(handle, p.n, N.ptr(p.f64), N.ptr(p.i32), len(p.pool), N.ptr(p.pool),
                                      N.ptr(p.pool_flag), p.probe)


@pytest.mark.parametrize("copies,bind", [(2, False), (40, False), (40, True)])
def test_triangulation_after_another_upload(copies, bind, native_lib):
    import torch
    surf = _surface(900, 3, 3.0)
    surf.getSurf(True, False, 0.0)
    area = surf.triangulateSurface()
    batch = nb.SurfaceBatch([surf] * copies)
    batch.getSurf()
    h = batch._context().handle
    if bind:
        p = surf.patches
        keep = [torch.from_numpy(a).cuda() for a in (p.f64, p.i32, p.pool, p.pool_flag)]
        torch.cuda.synchronize()
        N.check(N.lib().nsg_bind_patches_device(h, p.n, *[ctypes.c_void_p(t.data_ptr()) for t in keep[:2]],
                                                len(p.pool), *[ctypes.c_void_p(t.data_ptr()) for t in keep[2:]],
                                                p.probe), "bind")
    else:
        N.check(_upload(h, _surface(60, 1).patches), "upload")
    assert (batch.triangulateSurface() == area).all()
    assert batch.n_triangles == copies * len(surf.triangles)


def test_refused_batch_leaves_the_grid(native_lib):
    surf = _surface(300, 2)
    vol = surf.getSurf(True, False, 0.0)
    area = surf.triangulateSurface()
    h = surf.ctx.handle
    g = N.NsGrid()
    ctypes.pointer(g)[0] = surf.delphi.grid
    g.nx = g.ny = g.nz = 1200  # 1.44 M rays per set and structure
    n = 1500
    grids = (N.NsGrid * n)(*[g] * n)
    assert N.lib().nsg_set_batch(h, n, grids) == -4  # NSG_ERR_CAPACITY
    # what the cast left is still there, and the next cast runs on the same grid
    st = surf.delphi.status.copy()
    now = np.empty_like(st)
    N.check(N.lib().nsg_download_status(h, N.ptr(now)), "status")
    assert np.array_equal(now, st)
    v = ctypes.c_double()
    N.check(N.lib().nsg_raycast(h, N.STATUS | N.ACCURATE_TRIANGULATION, 0, ctypes.byref(v)), "raycast")
    assert v.value == vol
    assert surf.triangulateSurface() == area
