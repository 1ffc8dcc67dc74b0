"""Calls of one context in orders that a program may well make, although the Python classes do not.

* Patches uploaded or bound between a cast and its triangulation: the triangulation is that of the
  cast.
* A batch that is refused (more than 2^31 rays) leaves the grid before in force.
* A cast that fails (a ray with more hits than the overflow path holds) leaves no results: calls on
  the cast before it are refused, not answered from half-written arrays; the next cast is whole.
* Derivatives, normals and node maps of a cast are not read with patches of another number or a grid of
  another size: refused; with as many patches, or a grid of the same size, they are answered as before.
* An upload that fails for want of memory leaves no patches, and its error does not come back with the
  next call.
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


def test_failed_cast_leaves_no_results(native_lib):
    surf = _surface(327, 1)
    vol = surf.getSurf(True, True, 10.0, download=False)
    h = surf.ctx.handle
    n = 1100  # spheres within one another: 2,200 hits on the rays through their common centre
    f64, i32 = np.zeros((n, 20)), np.zeros((n, 4), np.int32)
    f64[:, 3] = 1.5 + 1e-4 * np.arange(n)
    g = surf.delphi.grid
    status = np.empty(g.nx * g.ny * g.nz, np.int32)
    ncav, area, v = ctypes.c_int(), ctypes.c_double(), ctypes.c_double()
    nv, nt = ctypes.c_int64(), ctypes.c_int64()
    flags = N.STATUS | N.ACCURATE_TRIANGULATION
    N.check(N.lib().nsg_upload_patches(h, n, N.ptr(f64), N.ptr(i32), 0, None, None, 1.4), "upload")
    assert N.lib().nsg_raycast(h, flags, 0, ctypes.byref(v)) == -4  # NSG_ERR_CAPACITY
    for rc in (N.lib().nsg_cavities(h, 10.0, ctypes.byref(ncav)), N.lib().nsg_download_status(h, N.ptr(status)),
               N.lib().nsg_triangulate(h, ctypes.byref(area), ctypes.byref(nv), ctypes.byref(nt)),
               N.lib().nsg_filter_cavities(h, 1.4, 0, None)):
        assert rc == -7  # NSG_ERR_STATE
    N.check(_upload(h, surf.patches), "upload")
    N.check(N.lib().nsg_raycast(h, flags, 0, ctypes.byref(v)), "raycast")
    N.check(N.lib().nsg_cavities(h, 10.0, ctypes.byref(ncav)), "cavities")
    assert v.value == vol and ncav.value > 0


def _read_all(h, n_patches, n_nodes, n_vertices):
    """Result codes of the calls that read a cast's arrays by patch or by node."""
    L = N.lib()
    eps, ideb = np.empty(3 * n_nodes, np.int32), np.empty(n_nodes, np.uint8)
    gv, normals = np.empty((n_patches, 8)), np.empty((n_vertices, 3))  # NSG_GRAD_PER_PATCH is 8
    n = ctypes.c_int64()
    by_patch = [L.nsg_patch_grads(h, N.ptr(gv), None), L.nsg_vertex_normals(h, N.ptr(normals))]
    by_node = [L.nsg_download_epsmap(h, N.ptr(eps)), L.nsg_download_idebmap(h, N.ptr(ideb)),
               L.nsg_bgp(h, 0, 50, ctypes.byref(n), None), L.nsg_filter_cavities(h, 1.4, 0, None)]
    return by_patch, by_node


def test_results_and_sizes_that_do_not_go_together(native_lib):
    L = N.lib()
    surf, other = _surface(327, 1), _surface(60, 1)
    surf.getSurf(True, False, 0.0)
    area = surf.triangulateSurface()
    h, g, p = surf.ctx.handle, surf.delphi.grid, surf.patches
    nodes = g.nx * g.ny * g.nz
    v, ncav, a = ctypes.c_double(), ctypes.c_int(), ctypes.c_double()
    nv, nt = ctypes.c_int64(), ctypes.c_int64()

    def cast():
        N.check(L.nsg_set_grid(h, ctypes.byref(g)), "grid")
        N.check(_upload(h, p), "upload")
        N.check(L.nsg_raycast(h, N.STATUS | N.ACCURATE_TRIANGULATION | N.EPSMAP | N.GRAD, 0, ctypes.byref(v)), "raycast")
        N.check(L.nsg_cavities(h, 10.0, ctypes.byref(ncav)), "cavities")

    def triangulate():
        N.check(L.nsg_triangulate(h, ctypes.byref(a), ctypes.byref(nv), ctypes.byref(nt)), "triangulate")

    cast()
    triangulate()
    assert _read_all(h, p.n, nodes, nv.value) == ([0, 0], [0, 0, 0, 0])
    # as many patches, the same grid
    cast()
    triangulate()
    N.check(_upload(h, p), "upload")
    N.check(L.nsg_set_grid(h, ctypes.byref(g)), "grid")
    assert _read_all(h, p.n, nodes, nv.value) == ([0, 0], [0, 0, 0, 0])
    # fewer patches: the cast's triangulation without its derivatives
    cast()
    N.check(_upload(h, other.patches), "upload")
    assert other.patches.n < p.n
    triangulate()
    assert nt.value > 0 and nv.value > 0
    assert _read_all(h, p.n, nodes, nv.value) == ([-7, -7], [0, 0, 0, 0])
    # a larger grid
    cast()
    triangulate()
    larger = _surface(900, 1).delphi.grid
    assert larger.nx > g.nx
    N.check(L.nsg_set_grid(h, ctypes.byref(larger)), "grid")
    assert _read_all(h, p.n, larger.nx * larger.ny * larger.nz, nv.value) == ([0, 0], [-7, -7, -7, -7])
    # and whole again
    cast()
    triangulate()
    assert _read_all(h, p.n, nodes, nv.value) == ([0, 0], [0, 0, 0, 0])
    assert area > 0


def test_failed_upload_leaves_no_patches(native_lib):
    L = N.lib()
    surf = _surface(327, 1)
    vol = surf.getSurf(True, False, 0.0)
    area = surf.triangulateSurface()
    h, p = surf.ctx.handle, surf.patches
    v, a = ctypes.c_double(), ctypes.c_double()
    nv, nt = ctypes.c_int64(), ctypes.c_int64()
    flags = N.STATUS | N.ACCURATE_TRIANGULATION | N.GRAD
    N.check(L.nsg_raycast(h, flags, 0, ctypes.byref(v)), "raycast")
    n = 1500 * 10**6  # 240 GB of records, refused before the host arrays are read
    assert L.nsg_upload_patches(h, n, N.ptr(p.f64), N.ptr(p.i32), 0, None, None, p.probe) < 0
    assert L.nsg_raycast(h, flags, 0, ctypes.byref(v)) == -7
    N.check(L.nsg_triangulate(h, ctypes.byref(a), ctypes.byref(nv), ctypes.byref(nt)), "triangulate")
    assert a.value == area  # the cast's, without derivatives
    gv = np.empty((p.n, 8))
    assert L.nsg_patch_grads(h, N.ptr(gv), None) == -7
    N.check(_upload(h, p), "upload")
    N.check(L.nsg_raycast(h, flags, 0, ctypes.byref(v)), "raycast")
    assert v.value == vol
