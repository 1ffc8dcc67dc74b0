"""Performance cases of the grid ray-casting surface builder.

Every case is one call sequence of a user's program: the whole molecule (``getSurf`` and
``triangulateSurface`` of the SES, skin or blobby surface), the differentiable volume and area, a
batch of conformers, a pipelined ensemble, pocket detection.  Molecules are the repository's seeded
globules (``generator.rsa_globule``); sizes, scales and options are those of its configurations,
tests and benchmark.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nanoshaper_b200 as nb
from nanoshaper_b200 import autograd
from nanoshaper_b200 import generator
from nanoshaper_b200.pipelined import PipelinedBatches


def listed():
    return [
        # the smallest molecule of the configurations (327 atoms, cavities filled up to 10 A^3): every
        # map and the mesh are brought back, as a desktop run does; all latency
        dict(name="ses_327", path="molecule", surface="ses", n=327, scale=2.0, perfil=70.0, precision="fp64",
             fill=10.0, eps=False, maps=True),
        # an ordinary protein at a fine grid, with cavities, maps and mesh
        dict(name="ses_2k", path="molecule", surface="ses", n=2000, scale=3.0, perfil=80.0, precision="fp64",
             fill=11.4, eps=False, maps=True),
        # the same size for a Poisson-Boltzmann solver: epsilon and ideb maps, boundary grid points
        # projected onto the surface
        dict(name="ses_eps_2k", path="molecule", surface="ses", n=2000, scale=2.0, perfil=80.0, precision="fp64",
             fill=10.0, eps=True, maps=True),
        # a large complex screened for volume, area and cavities: nothing dense comes back
        dict(name="ses_20k", path="molecule", surface="ses", n=20000, scale=4.0, perfil=70.0, precision="fp64",
             fill=11.4, eps=False, maps=False),
        # skin surface in mixed precision
        dict(name="skin_4k", path="molecule", surface="skin", n=4000, scale=3.0, perfil=80.0, precision="mixed",
             fill=-1.0, eps=False, maps=True),
        # blobby surface, its mesh built on the device in every pass
        dict(name="blobby_2k", path="molecule", surface="blobby", n=2000, scale=3.0, perfil=80.0, precision="fp64",
             fill=-1.0, eps=False, maps=True),
        # one gradient step of a torch program: forward and backward of volume and area
        dict(name="gradient_2k", path="gradient", surface="ses", n=2000, scale=3.0, perfil=80.0, precision="fp64"),
        dict(name="gradient_blobby_777", path="gradient", surface="blobby", n=777, scale=2.0, perfil=80.0,
             precision="mixed"),
        # fragments and peptides in one batch, volumes and areas in double precision
        dict(name="fragments_24", path="batch", bases=4, perturb=6, n_min=40, n_max=333, scale=2.0, perfil=80.0,
             precision="fp64", grad=False),
        # conformer ensemble of the benchmark (500 to 8,000 atoms) in mixed precision, with the atom
        # derivatives of every volume and area
        dict(name="conformers_64", path="batch", bases=4, perturb=16, n_min=500, n_max=8000, scale=2.0, perfil=80.0,
             precision="mixed", grad=True),
        # the same kind of ensemble from pinned host memory, copies overlapped with compute
        dict(name="pipelined_96", path="pipelined", bases=4, perturb=24, n_min=500, n_max=8000, scale=2.0,
             perfil=80.0, precision="mixed", chunks=8, contexts=4),
        # pockets by difference of a fat-probe and a small-probe cast
        dict(name="pockets_2k", path="pockets", n=2000, scale=2.0, perfil=80.0, precision="fp64"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    scale = round(rng.uniform(1.5, 3.2), 2)
    perfil = round(rng.uniform(68.0, 85.0), 1)
    precision = rng.choice(["fp64", "mixed"])
    path = rng.choice(["molecule", "molecule", "molecule", "gradient", "batch", "batch", "pipelined", "pockets"])
    if path == "molecule":
        surface = rng.choice(["ses", "ses", "skin", "blobby"])
        n = log_int(60, {"ses": 6000, "skin": 3500, "blobby": 1500}[surface])
        fill = rng.choice([-1.0, round(rng.uniform(5.0, 30.0), 1)])
        return dict(path=path, surface=surface, n=n, scale=min(scale, 2.6), perfil=perfil, precision=precision, fill=fill,
                    eps=surface == "ses" and n < 2500 and rng.random() < 0.4, maps=True)
    if path == "gradient":
        surface = rng.choice(["ses", "ses", "blobby"])
        return dict(path=path, surface=surface, n=log_int(60, 2500 if surface == "ses" else 800), scale=min(scale, 2.6),
                    perfil=perfil, precision=precision)
    if path == "pockets":
        return dict(path=path, n=log_int(200, 2500), scale=min(scale, 2.2), perfil=perfil, precision=precision)
    n_min = log_int(40, 900)
    case = dict(path=path, bases=rng.randint(1, 3), perturb=rng.randint(2, 12), n_min=n_min,
                n_max=n_min + log_int(50, 4000), scale=min(scale, 2.2), perfil=perfil, precision=precision)
    if path == "batch":
        case["grad"] = rng.random() < 0.5
    else:
        case["chunks"] = rng.randint(2, 6)
        case["contexts"] = rng.randint(1, 4)
    return case


# ---- what a program holds before the call ----

def _config(case, surface, probe=1.4):
    cf = nb.ConfigFile()
    cf.add("Surface", surface)
    cf.add("Probe_Radius", probe)
    cf.add("Accurate_Triangulation", True)
    cf.add("Triangulation", True)
    cf.add("Gpu_Precision", case["precision"])
    if case.get("eps"):
        cf.add("Project_boundary_grid_points", True)
    return cf


def _box(case):
    """The grid of a series of molecules of one size: that of the globule's bounding cube."""
    r = generator.globule_radius(case["n"]) + 1.8
    corners = np.array([[-r, -r, -r, 0.1], [r, r, r, 0.1]])
    return nb.DelPhiShared(corners, case["scale"], case["perfil"]).grid


def _surface(case, atoms, surface="ses", probe=1.4):
    ds = nb.DelPhiShared(atoms, case["scale"], case["perfil"], build_eps_map=bool(case.get("eps")),
                         grid=_box(case) if "n" in case else None)
    surf = nb.surfaceFactory().create(_config(case, surface, probe), ds)
    if surface != "blobby":
        surf.build()  # host patch construction, once per molecule
    return surf


def _ensemble(case, seed):
    rng = np.random.default_rng(seed)
    # the base sizes are spread over [n_min, n_max] in the same way for every seed
    sizes = np.round(np.linspace(case["n_min"], case["n_max"], case["bases"] + 1)[1:]).astype(int)
    nb.reset_seed()
    surfs = []
    for b, n in enumerate(sizes):
        base = generator.rsa_globule(int(n), seed=int(seed) * 64 + b)
        for _ in range(case["perturb"]):
            a = base.copy()
            a[:, :3] += rng.normal(0.0, 0.3, size=(len(a), 3))
            surfs.append(_surface(case, a))
    return surfs


def prepare(case, seed):
    path = case["path"]
    if path in ("batch", "pipelined"):
        surfs = _ensemble(case, seed)
        if path == "batch":
            return dict(case=case, batch=nb.SurfaceBatch(surfs))
        return dict(case=case, pipe=PipelinedBatches(surfs, n_chunks=case["chunks"], n_contexts=case["contexts"],
                                                     precision=case["precision"]))
    atoms = generator.rsa_globule(case["n"], int(seed))
    nb.reset_seed()
    if path == "molecule":
        return dict(case=case, surf=_surface(case, atoms, case["surface"]))
    if path == "pockets":
        fat = _surface(case, atoms, probe=3.0)
        nb.reset_seed()
        return dict(case=case, fat=fat, small=_surface(case, atoms, probe=1.4))
    t = torch.tensor(atoms, dtype=torch.float64)
    return dict(case=case, atoms=t, grid=autograd.grid_for(t, case["scale"], case["perfil"]))


# ---- the calls ----

def _kept(state, name, a, rows):
    """Result `a` (first axis of varying length) in the program's own array of `rows` rows, the rest
    zero, as a program that walks a series keeps it."""
    a = np.asarray(a)
    n = len(a)
    if n > rows:
        raise ValueError(f"{name}: {n} rows, {rows} kept")
    buf, used = state.get(name, (None, 0))
    if buf is None:
        buf = np.zeros((rows,) + a.shape[1:], a.dtype)
    buf[:n] = a
    buf[n:used] = 0
    state[name] = (buf, n)
    return buf


def _run_molecule(case, state):
    surf = state["surf"]
    n = case["n"]
    if case["surface"] == "blobby":
        surf.build()
    fill = case["fill"] >= 0.0
    out = {"volume": surf.getSurf(True, fill, max(case["fill"], 0.0), download=case["maps"])}
    out["area"] = surf.triangulateSurface(download=case["maps"])
    ds = surf.delphi
    if fill:
        out["cavity_sizes"] = _kept(state, "cavity_sizes", np.array(ds.cavitiesSize, np.float64), n + 100)
        out["cavity_filled"] = _kept(state, "cavity_filled", np.array(ds.cavitiesFlag, np.int32), n + 100)
        out["cavity_atoms"] = _kept(state, "cavity_atoms", np.array([a for cav in ds.cav2atoms for a in cav], np.int32),
                                    10 * n + 100)
    # skin and blobby surfaces of a globule have inner walls too
    rows = int((2.0 if case["surface"] == "ses" else 5.0) * _vertices(n, case["scale"])) + 2000
    if case["maps"]:
        out.update(status=ds.status, insideness=surf.insideness.view(np.int32),
                   vertices=_kept(state, "vertices", surf.vertices, rows),
                   triangles=_kept(state, "triangles", surf.triangles, 2 * rows))
    if case["eps"]:
        out.update(epsmap=ds.epsmap, idebmap=ds.idebmap, bgp=_kept(state, "bgp", ds.ibgp, rows),
                   bgp_pos=_kept(state, "bgp_pos", ds.scspos, rows), bgp_flag=_kept(state, "bgp_flag", ds.bgp_flag, rows))
    return out


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "molecule":
        return _run_molecule(case, state)
    if path == "gradient":
        atoms = state["atoms"].detach().requires_grad_()
        call = autograd.ses_volume_area if case["surface"] == "ses" else autograd.blobby_volume_area
        va = call(atoms, grid=state["grid"], precision=case["precision"])
        (va[0] + va[1]).backward()
        return {"volume": va.detach()[0], "area": va.detach()[1], "gradient": atoms.grad}
    if path == "batch":
        batch = state["batch"]
        out = {"volume": batch.getSurf(grad=case["grad"]), "area": batch.triangulateSurface()}
        if case["grad"]:
            g = batch.atom_gradients()
            out["gvol"] = np.concatenate([v for v, _ in g])
            out["garea"] = np.concatenate([a for _, a in g])
        return out
    if path == "pipelined":
        pipe = state["pipe"]
        vol, area = pipe.run()
        g = pipe.gradients()
        return {"volume": vol, "area": area, "gvol": np.concatenate([v for v, _ in g]),
                "garea": np.concatenate([a for _, a in g])}
    fat, small = state["fat"], state["small"]
    vols = [fat.getSurf(True, False, 0.0, download=False), small.getSurf(True, False, 0.0, download=False)]
    n = fat.difference(small, 0.0)
    return {"volume": np.array(vols), "pockets": n,
            "sizes": _kept(state, "sizes", np.array(fat.delphi.cavitiesSize, np.float64), 10 * case["n"] + 100),
            "status": fat.delphi.status, "insideness": fat.insideness.view(np.int32)}


# ---- what a pass cannot do without ----

def _vertices(n, scale):
    """Mesh vertices of a globule of n atoms: 3.6 scale^2 per SES patch, 20 n^0.72 patches."""
    return 3.6 * scale * scale * 20.0 * n ** 0.72


def _one(case, n, sets, grad):
    """Bytes and flops of one structure: patches in, candidates tested, results out.  The counts
    are those of the generator's globules: 20 n^0.72 SES patches with 5 pool entries each, and
    8.5 scale^2 candidate rays per patch and ray set."""
    surface = case.get("surface", "ses")
    scale = case["scale"]
    ses = 20.0 * n ** 0.72
    patches = {"ses": ses, "skin": 24.0 * n, "blobby": 7.0 * ses * scale * scale}[surface]
    verts = _vertices(n, scale)
    nodes = (200.0 / case["perfil"] * (1.37 * (36.0 * n / (4.0 * math.pi)) ** (1.0 / 3.0) + 1.7) * scale) ** 3
    data = 350.0 * patches if surface != "blobby" else 32.0 * n
    if case.get("maps"):
        data += 4.125 * nodes + 52.0 * verts + 24.0 * verts
    if case.get("eps"):
        data += 13.0 * nodes
    if grad:
        data += 64.0 * n
    flops = 130.0 * sets * 8.5 * scale * scale * ses * (2.0 if grad else 1.0) + 40.0 * verts
    if surface == "blobby":
        flops += n * (12.0 * scale) ** 3 * 30.0
    return data, flops


def work(case):
    path = case["path"]
    if path in ("batch", "pipelined"):
        grad = case.get("grad", True)
        sizes = np.linspace(case["n_min"], case["n_max"], case["bases"] + 1)[1:]
        parts = [_one(case, float(n), 4, grad) for n in sizes]
        return {"bytes": case["perturb"] * sum(p[0] for p in parts), "flops": case["perturb"] * sum(p[1] for p in parts)}
    if path == "pockets":
        d, f = _one(dict(case, maps=True), case["n"], 4, False)
        return {"bytes": d, "flops": 2.0 * f}
    d, f = _one(case, case["n"], 6 if case.get("eps") else 4, path == "gradient")
    return {"bytes": d, "flops": f}


def tolerance(case):
    # Sums of double-precision terms in another order differ by 1e-15 to 1e-13.  Mixed precision
    # refines FP32 roots to 1e-9 A by design, so that another correct refinement of a hit moves
    # positions by that much; labels, bits, edge codes and indices stay the same.
    if case["precision"] == "mixed":
        return {"rel": 1e-9, "max": 1e-8, "differ": 0.0}
    return {"rel": 1e-11, "max": 1e-9, "differ": 0.0}


# ---- the volume in 64 bits, ray by ray, in plain torch ----

_AXES = ((1, 2, 0), (0, 1, 2), (0, 2, 1))  # pixel axes and ray axis of the x, z and y panels


def _candidates(lo, hi, g, fd, ld, delta):
    """(patch, pixel, pixel) of every ray inside a patch's box, box corners given per patch."""
    mn = (g.xmin, g.ymin, g.zmin)
    nn = (g.nx, g.ny, g.nz)
    rng = []
    for d in (fd, ld):
        a = torch.ceil((lo[:, d] - mn[d] - delta) / g.side).clamp(0, nn[d])
        b = torch.floor((hi[:, d] - mn[d] - delta) / g.side).clamp(-1, nn[d] - 1)
        rng.append((a.long(), (b - a + 1).clamp(min=0).long()))
    (m0, w), (n0, h) = rng
    cnt = w * h
    p = torch.repeat_interleave(torch.arange(len(cnt), device=cnt.device), cnt)
    k = torch.arange(len(p), device=cnt.device) - (torch.cumsum(cnt, 0) - cnt)[p]
    m, n = m0[p] + k % w[p], n0[p] + k // w[p]
    return p, m, n, mn[fd] + m * g.side + delta, mn[ld] + n * g.side + delta


def _quartic_real(c):
    """Real roots of x^4 + c0 x^3 + c1 x^2 + c2 x + c3 (Weierstrass iteration); others are NaN."""
    rad = 1.0 + c.abs().amax(1, keepdim=True)
    rad = torch.minimum(rad, 2.0 * torch.stack([c[:, i].abs() ** (1.0 / (i + 1)) for i in range(4)], 1).amax(1, keepdim=True) + 1e-9)
    z = rad * torch.tensor([0.4 + 0.9j], dtype=torch.complex128, device=c.device) ** torch.arange(4, device=c.device)
    cc = c.to(torch.complex128)
    for _ in range(60):
        for i in range(4):
            x = z[:, i]
            f = (((x + cc[:, 0]) * x + cc[:, 1]) * x + cc[:, 2]) * x + cc[:, 3]
            d = torch.ones_like(x)
            for j in range(4):
                if j != i:
                    d = d * (x - z[:, j])
            z[:, i] = x - f / torch.where(d == 0, torch.full_like(d, 1e-30), d)
    x = torch.where(z.imag.abs() < 1e-6 * (1.0 + z.real.abs()), z.real, torch.full_like(z.real, float("nan")))
    a, b, e, f0 = (c[:, i:i + 1] for i in range(4))
    for _ in range(3):
        f = (((x + a) * x + b) * x + e) * x + f0
        df = ((4.0 * x + 3.0 * a) * x + 2.0 * b) * x + e
        x = x - torch.where(df == 0, torch.zeros_like(f), f / df)
    return x


def _hits(P, kind, first, cnt, pool, flag, probe, u, v, fd, ld, vc):
    """Roots along the ray axis (absolute coordinates, one column each, NaN where none) of the
    surfaces of the patch records P and whether each is on the patch."""
    if kind == "skin":
        Q = P[:, 4:14]
        A = torch.stack([Q[:, [0, 4, 7]], Q[:, [4, 1, 5]], Q[:, [7, 5, 2]]], 1)
        b = Q[:, [9, 8, 6]]
        c0 = P[:, :3]
        o = c0.clone()
        o[:, fd], o[:, ld] = u, v
        Ao = torch.einsum("nij,nj->ni", A, o)
        qa, qb = A[:, vc, vc], Ao[:, vc] + b[:, vc]
        qc = (o * (Ao + 2.0 * b)).sum(1) + Q[:, 3]
        s = torch.sqrt(qb * qb - qa * qc)
        x = torch.stack([(-qb - s) / qa, (-qb + s) / qa], 1) + c0[:, vc:vc + 1]
    elif kind == "torus":
        inv = P[:, 9:18].reshape(-1, 3, 3)
        o = P[:, :3].clone()
        o[:, fd], o[:, ld] = u, v
        y = o - P[:, 4:7]
        R2 = P[:, 7] ** 2
        ax = inv[:, 2]
        k = (y * y).sum(1) + R2 - probe * probe
        yv, z0, zs = y[:, vc], (ax * y).sum(1), ax[:, vc]
        # (s^2 + 2 yv s + k)^2 - 4 R^2 (s^2 + 2 yv s + |y|^2 - (z0 + zs s)^2)
        c = torch.stack([4 * yv, 4 * yv * yv + 2 * k - 4 * R2 * (1 - zs * zs), 4 * yv * k - 8 * R2 * (yv - z0 * zs),
                         k * k - 4 * R2 * ((y * y).sum(1) - z0 * z0)], 1)
        s = _quartic_real(c)
        d2 = (u - P[:, fd]) ** 2 + (v - P[:, ld]) ** 2
        s = torch.where(s * s + d2[:, None] < (P[:, 3] ** 2)[:, None], s, torch.full_like(s, float("nan")))
        x = s + P[:, vc:vc + 1]
    else:
        s = torch.sqrt(P[:, 3] ** 2 - (u - P[:, fd]) ** 2 - (v - P[:, ld]) ** 2)
        x = torch.stack([P[:, vc] - s, P[:, vc] + s], 1)
    pt = torch.empty(x.shape + (3,), dtype=torch.float64, device=x.device)
    pt[..., fd], pt[..., ld], pt[..., vc] = u[:, None], v[:, None], x
    ok = torch.isfinite(x)
    if kind == "torus":
        ok &= ~((P[:, 8] >= 0)[:, None] & (((pt - P[:, None, 4:7]) ** 2).sum(-1) < (P[:, 8] ** 2)[:, None]))
        accepted = (cnt == 0)[:, None].expand_as(ok).clone()
    for q in range(0, int(cnt.max()) if len(cnt) else 0, 2 if kind == "torus" else 1):
        has = (q < cnt)[:, None]
        e = first + torch.where(q < cnt, torch.full_like(cnt, q), torch.zeros_like(cnt))
        e = e.clamp(max=len(pool) - 2)
        w = pool[e][:, None]
        if kind == "point":
            ok &= ~(has & (((pt - w[..., :3]) ** 2).sum(-1) < w[..., 3]))
            continue
        t0 = (w[..., :3] * pt).sum(-1) + w[..., 3]
        if kind != "torus":
            ok &= ~(has & (t0 > 0))
            continue
        w1 = pool[e + 1][:, None]
        t1 = (w1[..., :3] * pt).sum(-1) + w1[..., 3]
        accepted |= has & torch.where((flag[e] != 0)[:, None], (t0 <= 0) & (t1 <= 0), (t0 <= 0) | (t1 <= 0))
    return x, (ok & accepted if kind == "torus" else ok)


def _volume(patches, g, sets):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = torch.from_numpy(patches.f64).to(dev)
    i32 = torch.from_numpy(patches.i32).to(dev).long()
    pool = torch.cat([torch.from_numpy(patches.pool).to(dev), torch.zeros((2, 4), dtype=torch.float64, device=dev)])
    flag = torch.cat([torch.from_numpy(patches.pool_flag).to(dev), torch.zeros(2, dtype=torch.int8, device=dev)])
    total = 0.0
    for s in sets:
        fd, ld, vc = _AXES[0 if s == 0 else (s - 1 if s <= 3 else s - 3)]
        delta = 1e-10 - g.hside if 1 <= s <= 3 else 0.0
        nb_ = (g.nx, g.ny, g.nz)[fd]
        rays, xs = [], []
        for kind, codes in (("point", (0,)), ("torus", (1, 2)), ("face", (3, 4)), ("skin", (5, 6, 7, 8))):
            ids = torch.nonzero(sum((i32[:, 0] == c) for c in codes) > 0)[:, 0]
            for at in range(0, len(ids), 8192):
                sel = ids[at:at + 8192]
                P = f64[sel]
                lo, hi = (P[:, 14:17], P[:, 17:20]) if kind == "skin" else (P[:, :3] - P[:, 3:4], P[:, :3] + P[:, 3:4])
                p, m, n, u, v = _candidates(lo, hi, g, fd, ld, delta)
                keep = (u - P[p, fd]) ** 2 + (v - P[p, ld]) ** 2 <= P[p, 3] ** 2
                if kind == "skin":
                    keep |= i32[sel[p], 0] != 5
                p, m, n, u, v = (t[keep] for t in (p, m, n, u, v))
                x, ok = _hits(P[p], kind, i32[sel[p], 1], i32[sel[p], 2], pool, flag, patches.probe, u, v, fd, ld, vc)
                r = (n * nb_ + m)[:, None].expand_as(x)
                rays.append(r[ok])
                xs.append(x[ok])
        r, x = torch.cat(rays), torch.cat(xs)
        x, order = torch.sort(x)
        r, order = torch.sort(r[order], stable=True)
        x = x[order]
        # interval lengths: +/- by position in the ray; rays with an odd number of hits are skipped
        _, inverse, count = torch.unique_consecutive(r, return_inverse=True, return_counts=True)
        start = torch.cumsum(count, 0) - count
        even = (torch.arange(len(r), device=dev) - start[inverse]) % 2 == 0
        good = count[inverse] % 2 == 0
        total += float((torch.where(even, -x, x) * good).sum())
    return g.A * total / len(sets)


def exact(case, seed):
    """The volume from the patch set by ray casting in plain torch; the area, the maps and the mesh
    follow from the same interval ends.  None for the surfaces without an analytic patch set and for
    the differentiable calls, which build their patches inside."""
    path = case["path"]
    if path in ("batch", "pipelined"):
        if case["perturb"] * case["bases"] * case["n_max"] > 150000:
            return None
        return {"volume": np.array([_volume(s.patches, s.delphi.grid, range(4)) for s in _ensemble(case, seed)])}
    if path == "gradient" or case.get("surface") == "blobby":
        return None
    state = prepare(case, seed)
    if path == "pockets":
        return {"volume": np.array([_volume(state[k].patches, state[k].delphi.grid, range(4)) for k in ("fat", "small")])}
    surf = state["surf"]
    return {"volume": _volume(surf.patches, surf.delphi.grid, range(6) if case["eps"] else range(4))}
