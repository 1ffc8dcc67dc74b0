"""The one-pass kernels (look-back offsets), their tickets and capacities, and the shared state of
the contexts.

* Overflow rays (50 hits) along each axis, next to ordinary ones, against the oracle: the vertex
  pass's per-lane path.
* Grids whose active-cube map and rays fill a 256-item ticket exactly, miss it or exceed it by a
  little, against the oracle.
* A batch of one structure 1, 9 and 70 times over, which crosses the 4-item and 8-item tickets:
  every copy's mesh, volume and area equal the single run's bit for bit.
* A triangulation of pockets, whose edges carry no analytic vertex, so that the first capacities do
  not suffice: triangle and vertex counts from the downloaded bits and the case table.
* Boundary grid points of grids below one ticket and of lattices whose points exceed the first
  capacity, against their definition in NumPy.
* Contexts one after another, in threads at the same time, and after nsg_release_kept give the
  same results.
"""
import ctypes
import threading
from pathlib import Path

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


def _surface(atoms, scale, perfil=80.0, probe=1.4, precision="fp64", grid=None):
    nb.reset_seed()
    cf = nb.ConfigFile(text=f"Surface = ses\nProbe_Radius = {probe}\nAccurate_Triangulation = true\n"
                            f"Triangulation = true\nGpu_Precision = {precision}\n")
    surf = nb.surfaceFactory().create(cf, nb.DelPhiShared(atoms, scale, perfil, grid=grid))
    surf.build()
    return surf


def _against_oracle(surf, oracle_mod, cav_vol=10.0):
    import compare
    surf.getSurf(True, True, cav_vol, keep_hits=True)
    surf.triangulateSurface()
    ref = oracle_mod.run(surf.delphi.grid, surf.patches, cav_vol=cav_vol)
    compare.compare_surface(surf, surf.delphi, ref)
    return ref


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_overflow_rays(axis, native_lib, oracle_mod):
    atoms = np.zeros((26, 4))
    atoms[:25, axis] = 6.5 * np.arange(25) - 78.0  # isolated spheres: two hits each
    atoms[25, (axis + 1) % 3] = 5.0
    atoms[:, 3] = 1.7
    surf = _surface(atoms, 1.0, 90.0)
    _against_oracle(surf, oracle_mod)
    assert surf.stats()["overflow_rays"] > 0


@pytest.mark.parametrize("nx,ny,nz", [(34, 18, 18), (34, 19, 18), (35, 18, 18), (66, 34, 34), (33, 35, 16), (16, 16, 16),
                                      (17, 16, 15), (97, 24, 33)])
def test_ticket_edges(nx, ny, nz, native_lib, oracle_mod):
    """(nx-2+31)/32 * (ny-2) * (nz-2) map words: 256 for the first grid, then one row more, a second
    word per row, exact multiples, and grids whose rays end inside a ticket."""
    atoms = np.array([[0.3, -0.2, 0.1, 1.7], [1.9, 0.4, -0.6, 1.5], [-0.8, 1.7, 0.9, 1.6]])
    g = N.NsGrid()
    ctypes.pointer(g)[0] = nb.DelPhiShared(atoms, 2.0, 50.0).grid
    side = 10.0 / min(nx, ny, nz)
    g.nx, g.ny, g.nz = nx, ny, nz
    g.scale, g.side, g.hside, g.A = 1.0 / side, side, 0.5 * side, side * side
    for n, lo, hi in ((nx, "xmin", "xmax"), (ny, "ymin", "ymax"), (nz, "zmin", "zmax")):
        half = 0.5 * (n - 1) * side
        setattr(g, lo, -half)
        setattr(g, hi, half)
    _against_oracle(_surface(atoms, 2.0, grid=g), oracle_mod)


@pytest.mark.parametrize("cells,scale", [(1, 2.0), (2, 2.0), (4, 1.0), (20, 1.0)])
def test_boundary_points(cells, scale, native_lib):
    """Spheres of 1.5 on a lattice of 3.6: most nodes have codes that differ, so that the largest
    grid has more points than a sixteenth of its nodes and the pass runs a second time."""
    c = 3.6 * np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    surf = _surface(np.concatenate([c, np.full((len(c), 1), 1.5)], 1), scale, 85.0, probe=0.3)
    ds = surf.delphi
    ds.buildEpsMap = True
    surf.projBGP = True
    surf.getSurf(True, False, 0.0)
    e = ds.epsmap
    codes = np.stack([e[1:, 1:, 1:, 0], e[1:, 1:, 1:, 1], e[1:, 1:, 1:, 2], e[1:, 1:, :-1, 0], e[1:, :-1, 1:, 1],
                      e[:-1, 1:, 1:, 2]])
    differ = (codes != codes[0]).any(0)
    kji = np.argwhere(differ) + 1
    assert np.array_equal(ds.ibgp, kji[:, ::-1])
    assert np.array_equal(ds.bgp_type == 1, (codes == 0).any(0)[differ])
    assert ds.nbgp > 0 and (ds.nbgp > e[..., 0].size / 16 + 4096) == (cells == 20)


@pytest.mark.parametrize("copies,precision", [(1, "fp64"), (9, "mixed"), (70, "fp64")])
def test_batch_copies_equal_single(copies, precision, native_lib):
    surf = _surface(generator.rsa_globule(900, 3), 3.0, precision=precision)
    vol = surf.getSurf(True, False, 0.0)
    area = surf.triangulateSurface()
    st = surf.stats()
    na, nt = st["analytic_vertices"], st["triangles"]
    nm = st["vertices"] - na
    batch = nb.SurfaceBatch([surf] * copies)
    assert (batch.getSurf(download=True) == vol).all()
    assert (batch.triangulateSurface() == area).all()
    assert batch.n_vertices == copies * (na + nm) and batch.n_triangles == copies * nt
    for bits in batch.insideness:
        assert np.array_equal(bits, surf.insideness)
    v = np.empty((batch.n_vertices, 3))
    t = np.empty((batch.n_triangles, 3), np.int32)
    N.check(N.lib().nsg_download_mesh(batch._context().handle, N.ptr(v), None, N.ptr(t)), "mesh")
    for b in range(copies):
        assert np.array_equal(v[b * na:(b + 1) * na], surf.vertices[:na])
        mid0 = copies * na + b * nm
        assert np.array_equal(v[mid0:mid0 + nm], surf.vertices[na:])
        tb = surf.triangles.astype(np.int64)
        tb = np.where(tb < na, tb + b * na, tb - na + mid0)
        assert np.array_equal(t[b * nt:(b + 1) * nt], tb)


def test_capacities_of_a_mesh_of_midpoints(native_lib):
    atoms = generator.rsa_globule(1500, 5)
    fat, small = _surface(atoms, 2.0, probe=3.0), _surface(atoms, 2.0, probe=1.4)
    for s in (fat, small):
        s.getSurf(True, False, 0.0, download=False)
    assert fat.difference(small, 0.0) > 0
    fat.triangulateSurface()
    g = fat.delphi.grid
    bits = np.unpackbits(fat.insideness.view(np.uint8), bitorder="little")[:g.nx * g.ny * g.nz]
    inside = bits.reshape(g.nz, g.ny, g.nx) == 0
    # corners of cube (i, j, k) in the table's order, cubes 1..n-2 of each axis
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    case = np.zeros((g.nz - 2, g.ny - 2, g.nx - 2), np.int64)
    for q, (dx, dy, dz) in enumerate(corner):
        case |= inside[1 + dz:g.nz - 1 + dz, 1 + dy:g.ny - 1 + dy, 1 + dx:g.nx - 1 + dx].astype(np.int64) << q
    table = np.load(ROOT / "tests" / "golden" / "fixtures" / "mc_tritable.npy")
    n_tri = (table.reshape(256, -1) >= 0).sum(1) // 3
    for face in (case[0], case[:, 0], case[:, :, 0]):  # no low-face cubes, which may lack vertices
        assert np.isin(face, (0, 255)).all()
    assert len(fat.triangles) == n_tri[case].sum()
    assert fat.triangles.min() >= 0 and fat.triangles.max() < len(fat.vertices)
    # a vertex per cut edge of the cube range, or more (two pair ends on one edge)
    own = [(5, 6), (6, 7), (2, 6)]
    cut = sum((((case >> a) ^ (case >> b)) & 1).sum() for a, b in own)
    assert len(fat.vertices) >= cut
    st = fat.stats()
    assert st["vertices"] - st["analytic_vertices"] > st["analytic_vertices"]  # mostly midpoints
    # and once more, with the ratios that the first run left
    again = fat.triangles.copy()
    fat.triangulateSurface()
    assert np.array_equal(again, fat.triangles)


def test_contexts_share_kept_memory(native_lib):
    def run(seed):
        surf = _surface_locked(seed)
        vol = surf.getSurf(True, True, 10.0)
        area = surf.triangulateSurface()
        out = (vol, area, surf.delphi.status.copy(), surf.triangles.copy(), [list(a) for a in surf.delphi.cav2atoms])
        surf.ctx.close()
        return out

    lock = threading.Lock()  # the jitter generator is one per process

    def _surface_locked(seed):
        with lock:
            return _surface(generator.rsa_globule(300 + 40 * seed, seed), 3.0)

    def same(a, b):
        return a[:2] == b[:2] and np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3]) and a[4] == b[4]

    first = [run(s) for s in range(4)]
    assert all(same(run(s), first[s]) for s in range(4))
    got = [None] * 4
    threads = [threading.Thread(target=lambda s=s: got.__setitem__(s, run(s))) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(g is not None and same(g, first[s]) for s, g in enumerate(got))
    N.release_kept()
    assert all(same(run(s), first[s]) for s in range(4))
