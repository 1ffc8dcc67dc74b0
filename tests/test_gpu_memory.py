"""Device memory that the library keeps from one context to the next.

* Beside live contexts that hold more than 8 GiB, the memory of a context that ends is kept for the next
  one, and nothing goes back to the driver within other calls.
* What is kept stays within a sixteenth of the memory that is free otherwise (or 512 MiB), so that other
  allocators of the process find the rest; nsg_release_kept gives back all of it.
"""
import gc

import numpy as np
import pytest

import nanoshaper_b200 as nb
from nanoshaper_b200 import _native as N
from nanoshaper_b200 import generator

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _surface(atoms, scale, perfil):
    nb.reset_seed()
    cf = nb.ConfigFile(text="Surface = ses\nProbe_Radius = 1.4\nAccurate_Triangulation = true\nTriangulation = true\n")
    surf = nb.surfaceFactory().create(cf, nb.DelPhiShared(atoms, scale, perfil))
    surf.build()
    return surf


def _large():
    """A few atoms on a grid of some 1,000^3 nodes: a context of more than 1.5 GiB."""
    atoms = np.array([[0.0, 0.0, 0.0, 1.7], [2.1, 0.4, -0.3, 1.5], [-40.0, -40.0, -40.0, 1.6], [40.0, 40.0, 40.0, 1.6]])
    return _surface(atoms, 11.0, 90.0)


def _run(surf):
    surf.getSurf(True, False, 0.0, download=False)
    return surf.volume, surf.triangulateSurface(download=False)


def test_kept_beside_large_contexts(native_lib):
    import torch
    torch.zeros(1, device="cuda")
    gc.collect()  # contexts that other tests left
    N.release_kept()
    before = _free()
    live = [_large()]
    want = _run(live[0])
    while before - _free() < 9 << 30:
        live.append(_large())
        assert _run(live[-1]) == want
    small = _surface(generator.rsa_globule(2000, 3), 2.0, 80.0)
    first = _run(small)
    with_small = _free()
    for _ in range(3):
        small.ctx.close()
        small.ctx = None
        assert _run(live[0]) == want  # waits often
        assert _free() == with_small  # neither given back ...
        assert _run(small) == first
        assert _free() == with_small  # ... nor mapped anew
    for s in live + [small]:
        s.ctx.close()
    N.release_kept()
    assert _free() > before - 64 * MIB


@pytest.mark.parametrize("left_gib", [3, 20])
def test_kept_is_a_share_of_what_is_free(left_gib, native_lib):
    import torch
    torch.zeros(1, device="cuda")
    gc.collect()
    N.release_kept()
    others = torch.empty(_free() - (left_gib << 30), dtype=torch.uint8, device="cuda")
    before = _free()
    surf = _large()
    _run(surf)
    assert before - _free() > 1536 * MIB
    surf.ctx.close()
    kept = before - _free()
    assert 0 < kept <= max(512 * MIB, before / 16) + 64 * MIB  # and what a pool cannot give back of a chunk
    N.release_kept()
    assert _free() > before - 64 * MIB
    del others
    torch.cuda.empty_cache()
