"""The single-precision screen of torus candidates on the GPU: the same casts with the screen off, on and
chosen by size give the same hits on every ray, bit for bit, the same volume and the same pairs, in both
precisions; small and large sets (below and above the line from which it is used), dense and loose
globules, small and large probes, sizes at which its distance test is left out."""
import ctypes

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

pytestmark = pytest.mark.gpu


def _cast(surf, screen):
    L, h = N.lib(), surf._context().handle
    p = np.zeros(6, np.int32)
    N.check(L.nsg_get_tuning(h, N.ptr(p), 6), "get tuning")
    p[4] = screen
    N.check(L.nsg_set_tuning(h, N.ptr(p), 6), "set tuning")
    vol = surf.getSurf(True, False, 0.0, keep_hits=True)
    launches = L.nsg_launch_count(h)
    surf.getSurf(True, False, 0.0, keep_hits=True)
    launches = L.nsg_launch_count(h) - launches
    g = surf.delphi.grid
    out = [np.array(vol)]
    for ray_set, n_rays in ((0, g.ny * g.nz), (1, g.ny * g.nz), (2, g.nx * g.ny), (3, g.nx * g.nz)):
        counts = np.zeros(n_rays, np.int32)
        total = L.nsg_download_hits(h, ray_set, N.ptr(counts), None, 0)
        hits = np.empty(total)
        N.check(L.nsg_download_hits(h, ray_set, N.ptr(counts), N.ptr(hits), total), "hits")
        out += [counts, hits]
    area = surf.triangulateSurface()
    return out + [np.array(area), surf.vertices.copy(), surf.triangles.copy()], launches


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,probe,scale,inflate,unit", [
    (40, 1.4, 2.0, 1.37, 1.0), (327, 1.4, 2.0, 1.37, 1.0), (3000, 1.4, 2.5, 1.37, 1.0), (600, 0.5, 3.0, 1.6, 1.0),
    (800, 3.0, 3.0, 1.37, 1.0), (500, 5.0, 2.5, 2.2, 1.0), (500, 1.4, 2.5, 1.37, 0.1), (500, 1.4, 2.5, 1.37, 10.0)])
def test_screen_changes_no_hit(n, probe, scale, inflate, unit, precision, native_lib):
    atoms = generator.rsa_globule(n, n, inflate=inflate) * unit
    nb.reset_seed()
    cf = nb.ConfigFile(text=f"Surface = ses\nProbe_Radius = {probe * unit}\nAccurate_Triangulation = true\n"
                            f"Triangulation = true\nGpu_Precision = {precision}\n")
    surf = nb.surfaceFactory().create(cf, nb.DelPhiShared(atoms, scale / unit, 80.0))
    surf.build()
    off, launches_off = _cast(surf, 1)
    on, launches_on = _cast(surf, 2)
    auto, launches_auto = _cast(surf, 0)
    assert launches_on == launches_off + 1  # the screen is one launch for all ray sets
    if n in (40, 3000):  # below and above the line
        assert launches_auto == (launches_off if n == 40 else launches_on)
    assert off[0] > 0 and off[1].sum() > 0
    for a, b, c in zip(off, on, auto):
        assert np.array_equal(a, b) and np.array_equal(a, c)
