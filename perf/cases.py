"""The work a user of this package has it do, as measurable cases.

Each case is a dict of plain values whose ``kind`` names the call:

* ``query``   closest points of a mesh that is built already: ``MeshBVH.udf``,
              ``MeshBVH.sdf`` (pseudo-normal sign);
* ``adjoint`` signed distances forward and their gradients w.r.t. points and
              mesh vertices (shape fitting);
* ``rebuild`` a new ``MeshBVH`` from moved vertices and one query of it (one
              step of a deforming-mesh loop: build and query);
* ``batch``   ``BatchedMeshBVH``: build and query of many uneven meshes;
* ``rays``    ``MeshBVH.intersect_ray``, nearest hit;
* ``parity``  ``MeshBVH.sdf(mode="parity")`` (meshes whose normals are not to
              be trusted);
* ``flood``   ``sparse_flood_fill`` and ``construct_surface_dual_graph``:
              mesh to labelled voxels to the extraction grid;
* ``clip``    ``OctreeIndexer.octree_traverse`` to the finest level, then
              ``MeshBVH.intersect_aabb(mode=3)`` on its cubes;
* ``dmc``     ``SparseDiffDMC``: training step (forward and backward) or the
              QEF inference forward.

Sizes come from the package's benchmark and tests: 20,480- to
1,310,720-triangle displaced spheres, 100,000 to 16,777,216 queries, octrees
to 1024^3, dual marching cubes to 512^3.  ``draw`` spreads over the same
ranges with tori of any triangle count besides the spheres, rough surfaces,
stretched meshes and odd sizes.  Inputs come from the case and the seed.
"""

from __future__ import annotations

import math

import torch

from atom3d_b200 import MeshBVH, OctreeIndexer, SparseDiffDMC, sparse_flood_fill, synthetic
from atom3d_b200.apps import construct_surface_dual_graph
from atom3d_b200.batch import BatchedMeshBVH
from atom3d_b200.mesh_extractor.dmc_tables import table

DEV = "cuda"
F64 = torch.float64
# point-triangle pairs the 64-bit brute force takes in about 15 seconds
EXACT_PAIRS = 2.6e10


def listed():
    return [
        # interactive signed-distance probe: a thousand points, launch bound
        {"name": "sdf_points_1k", "kind": "query", "shape": "sphere", "tris": 20480, "rough": True, "stretch": 1.0,
         "points": 1021, "signed": True},
        # the test suite's first workload: 100,000 points, 20,480 triangles
        {"name": "udf_100k", "kind": "query", "shape": "sphere", "tris": 20480, "rough": True, "stretch": 1.0,
         "points": 100000, "signed": False},
        # the benchmark's headline: distance-field sampling of a large scan
        {"name": "udf_16m", "kind": "query", "shape": "sphere", "tris": 1310720, "rough": False, "stretch": 1.0,
         "points": 16777216, "signed": False},
        # one gradient step of fitting a mesh to signed-distance samples
        {"name": "sdf_grad_300k", "kind": "adjoint", "shape": "sphere", "tris": 81920, "rough": False,
         "stretch": 1.0, "points": 300007},
        # deforming mesh: new tree every step, a modest number of samples
        {"name": "rebuild_1m_tris", "kind": "rebuild", "shape": "sphere", "tris": 1310720, "rough": False,
         "stretch": 1.0, "points": 262144},
        # data preparation over a set of meshes of uneven size
        {"name": "batch_24", "kind": "batch", "meshes": 24, "min_level": 3, "max_level": 7, "per_tri": 4},
        # camera and scattered rays against a large scan
        {"name": "rays_4m", "kind": "rays", "shape": "sphere", "tris": 1310720, "rough": False, "stretch": 1.0,
         "rays": 4194304},
        # inside/outside by ray parity, eight directions a point
        {"name": "parity_100k", "kind": "parity", "shape": "torus", "tris": 200000, "rough": False, "stretch": 1.0,
         "points": 100003, "dirs": 8},
        # mesh to labelled 1024^3 voxels and the dual graph of its surface cells
        {"name": "flood_1024", "kind": "flood", "shape": "sphere", "tris": 327680, "rough": False, "stretch": 1.0,
         "level": 10, "connectivity": 26},
        # voxelisation with the clipped polygons of every (cube, face) pair
        {"name": "clip_512", "kind": "clip", "shape": "sphere", "tris": 327680, "rough": False, "stretch": 1.0,
         "level": 9},
        # training step of the differentiable extraction at 512^3
        {"name": "dmc_train_512", "kind": "dmc", "res": 512, "spheres": 32, "mode": "train", "weights": False},
        # inference extraction at an odd, moderate resolution
        {"name": "dmc_qef_200", "kind": "dmc", "res": 200, "spheres": 12, "mode": "qef", "weights": True},
    ]


def _spread(rng, lo, hi):
    """Log-uniform whole number in [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_mesh(rng, lo, hi):
    stretch = rng.choice([1.0, 1.0, round(rng.uniform(0.4, 2.5), 2)])
    rough = rng.random() < 0.3
    if rng.random() < 0.5:
        sizes = [t for t in (20 * 4 ** k for k in range(2, 9)) if lo <= t <= hi]
        return {"shape": "sphere", "tris": rng.choice(sizes), "rough": rough, "stretch": stretch}
    return {"shape": "torus", "tris": _spread(rng, lo, hi), "rough": rough, "stretch": stretch}


def draw(rng):
    kind = rng.choice(["query", "query", "query", "adjoint", "rebuild", "batch", "rays", "parity", "flood", "clip",
                       "dmc", "dmc"])
    c = {"kind": kind}
    if kind == "query":
        c.update(_draw_mesh(rng, 320, 1310720))
        c.update(points=_spread(rng, 500, 8000000), signed=rng.random() < 0.5)
    elif kind == "adjoint":
        c.update(_draw_mesh(rng, 1280, 327680))
        c.update(points=_spread(rng, 2000, 1000000))
    elif kind == "rebuild":
        c.update(_draw_mesh(rng, 320, 1310720))
        c.update(points=_spread(rng, 1000, 300000))
    elif kind == "batch":
        c.update(meshes=rng.randint(2, 40), min_level=rng.randint(2, 3), max_level=rng.randint(4, 6),
                 per_tri=rng.randint(1, 8))
    elif kind == "rays":
        c.update(_draw_mesh(rng, 320, 1310720))
        c.update(rays=_spread(rng, 1000, 8000000))
    elif kind == "parity":
        c.update(_draw_mesh(rng, 1280, 327680))
        c.update(points=_spread(rng, 1000, 300000), dirs=rng.choice([4, 8]))
    elif kind in ("flood", "clip"):
        c.update(_draw_mesh(rng, 1280, 327680))
        c.update(level=rng.randint(6, 9))
        if kind == "flood":
            c.update(connectivity=rng.choice([6, 26]))
    else:
        c.update(res=_spread(rng, 24, 480), spheres=rng.randint(2, 32), mode=rng.choice(["train", "train", "qef"]),
                 weights=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_ICO = {}


def _icosphere(tris):
    level = 0
    while 20 * 4 ** level < tris:
        level += 1
    if level not in _ICO:
        _ICO[level] = synthetic.icosphere(level)
    v, f = _ICO[level]
    return v.to(DEV).double(), f.to(DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _bumps(x, g, terms=16, amp=0.05):
    """Sum of seeded sinusoids over unit directions x."""
    freq = torch.rand(terms, generator=g, dtype=F64, device=DEV) * 6.0 + 2.0
    d = torch.randn(terms, 3, generator=g, dtype=F64, device=DEV)
    d = d / d.norm(dim=1, keepdim=True)
    ph = torch.rand(terms, generator=g, dtype=F64, device=DEV) * (2 * math.pi)
    s = torch.zeros(x.shape[0], dtype=F64, device=DEV)
    for k in range(terms):
        s += torch.sin(freq[k] * (x * d[k]).sum(1) + ph[k])
    return amp * s


def _mesh(case, g):
    """(vertices float32 [V,3], faces int32 [F,3]) of a closed, outward surface."""
    if case["shape"] == "sphere":
        x, f = _icosphere(case["tris"])
        v = x * (1.0 + _bumps(x, g))[:, None]
    else:
        nv = max(4, int(math.sqrt(case["tris"] / 6.0)))
        nu = max(4, case["tris"] // (2 * nv))
        u = torch.arange(nu, device=DEV, dtype=F64) * (2 * math.pi / nu)
        w = torch.arange(nv, device=DEV, dtype=F64) * (2 * math.pi / nv)
        uu, ww = torch.meshgrid(u, w, indexing="ij")
        n = torch.stack([torch.cos(uu) * torch.cos(ww), torch.sin(uu) * torch.cos(ww), torch.sin(ww)], -1).reshape(-1, 3)
        c = torch.stack([torch.cos(uu), torch.sin(uu), torch.zeros_like(uu)], -1).reshape(-1, 3) * 0.9
        v = c + n * (0.4 * (1.0 + _bumps(n, g, 6, 0.03)))[:, None]
        i = torch.arange(nu, device=DEV)[:, None].expand(nu, nv)
        j = torch.arange(nv, device=DEV)[None].expand(nu, nv)
        i1, j1 = (i + 1) % nu, (j + 1) % nv
        a, b, cc, d = i * nv + j, i1 * nv + j, i1 * nv + j1, i * nv + j1
        f = torch.stack([torch.stack([a, b, cc], -1), torch.stack([a, cc, d], -1)], 2).reshape(-1, 3).int()
    if case["rough"]:
        edge = 2.0 / math.sqrt(f.shape[0] / 5.0)
        v = v * (1.0 + 0.25 * edge * torch.randn(v.shape[0], generator=g, dtype=F64, device=DEV))[:, None]
    v = v * torch.tensor([case["stretch"], 1.0, 1.0], dtype=F64, device=DEV)
    return v.float().contiguous(), f.contiguous()


def _samples(v, f, n, g, sigma=0.02, box_scale=1.2):
    """Half near the surface (a point of a random face + N(0, sigma)), half
    uniform in the mesh box scaled by ``box_scale``."""
    ns = n // 2
    vd = v.double()
    t = vd[f[torch.randint(0, f.shape[0], (ns,), generator=g, device=DEV)].long()]
    r = torch.rand(ns, 2, generator=g, dtype=F64, device=DEV)
    s = r[:, 0].sqrt()
    w = torch.stack([1 - s, s * (1 - r[:, 1]), s * r[:, 1]], 1)
    near = (w[:, :, None] * t).sum(1) + sigma * torch.randn(ns, 3, generator=g, dtype=F64, device=DEV)
    lo, hi = vd.min(0).values, vd.max(0).values
    u = torch.rand(n - ns, 3, generator=g, dtype=F64, device=DEV) * 2 - 1
    return torch.cat([near, (lo + hi) * 0.5 + u * (hi - lo) * (0.5 * box_scale)]).float()


def _mesh_points(case, seed):
    g = _gen(seed)
    v, f = _mesh(case, g)
    return v, f, _samples(v, f, case["points"], g)


def _mesh_rays(case, seed):
    """Half a pinhole camera's rays in scan order, half scattered ones."""
    g = _gen(seed)
    v, f = _mesh(case, g)
    n = case["rays"]
    nc = n // 2
    side = max(1, int(math.ceil(math.sqrt(nc))))
    k = torch.arange(nc, device=DEV)
    px = ((k % side).double() + 0.5) / side * 2 - 1
    py = ((k // side).double() + 0.5) / side * 2 - 1
    eye = torch.randn(3, generator=g, dtype=F64, device=DEV)
    eye = eye / eye.norm() * 4.0
    fwd = -eye / eye.norm()
    up = torch.tensor([0.3, 0.2, 1.0], dtype=F64, device=DEV)
    right = torch.linalg.cross(fwd, up)
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    dc = fwd + 0.45 * (px[:, None] * right + py[:, None] * up)
    lo, hi = v.double().min(0).values, v.double().max(0).values
    u = torch.rand(n - nc, 3, generator=g, dtype=F64, device=DEV) * 2 - 1
    os = (lo + hi) * 0.5 + u * (hi - lo) * 0.6
    ds = torch.randn(n - nc, 3, generator=g, dtype=F64, device=DEV)
    o = torch.cat([eye[None].expand(nc, 3), os])
    d = torch.cat([dc, ds])
    return v, f, o.float().contiguous(), (d / d.norm(dim=1, keepdim=True)).float().contiguous()


def _voxel_mesh(case, seed):
    """A mesh placed in the grid [-1, 1]^3 of 2^level cells a side.

    Its shape belongs to the case and its place to the seed: the vertices lie
    on a binary grid and move by whole cells, so every seed's voxels, labels
    and pairs are as many; the faces come in an order of the seed's own."""
    v, f = _mesh(case, _gen(case["tris"] + case["level"]))
    half = 1 << (case["level"] - 1)
    extent = min(0.9, 1.0 - 16.0 / half)  # room for the flood's 10-cell padding
    v = torch.round(v.double() * (extent / float(v.abs().max())) * 2.0 ** 21) / 2.0 ** 21
    g = _gen(seed)
    f = f[torch.randperm(f.shape[0], generator=g, device=DEV)]
    if case["kind"] == "flood":
        v = v + torch.randint(-4, 5, (3,), generator=g, device=DEV).double() / half
    return v.float().contiguous(), f.contiguous()


def _batch_inputs(case, seed):
    g = _gen(seed)
    meshes, pts, counts = [], [], []
    span = case["max_level"] - case["min_level"] + 1
    for i in range(case["meshes"]):
        level = case["min_level"] + i % span
        v, f = _mesh({"shape": "sphere", "tris": 20 * 4 ** level, "rough": False, "stretch": 1.0}, g)
        sc = torch.rand(1, generator=g, device=DEV) * 1.5 + 0.5
        v = (v * sc + torch.rand(3, generator=g, device=DEV) * 2 - 1).contiguous()
        meshes.append((v, f))
        p = _samples(v, f, case["per_tri"] * f.shape[0], g)
        pts.append(p)
        counts.append(p.shape[0])
    return meshes, torch.cat(pts), counts


def _dmc_inputs(case, seed):
    """Cubes of a [-1, 1]^3 grid in a band about a union of spheres, the
    noisy distances at their corners and, with weights, deform / alpha / beta.
    The cubes and the signs belong to the case, the values to the seed (as
    between two steps of a training run)."""
    res, k = case["res"], case["spheres"]
    g = _gen(1000 * res + k)
    ctr = torch.rand(k, 3, generator=g, dtype=F64, device=DEV) * 1.4 - 0.7
    rad = torch.rand(k, generator=g, dtype=F64, device=DEV) * 0.15 + 0.05
    h = 2.0 / res
    band = 2 * h + 0.5 * math.sqrt(3.0) * h

    def field(x):
        d = torch.full((x.shape[0],), float("inf"), dtype=F64, device=DEV)
        for i in range(k):
            d = torch.minimum(d, (x - ctr[i]).norm(dim=1) - rad[i])
        return d

    blk = 8
    nb = -(-res // blk)
    ax = torch.arange(nb, device=DEV)
    bi = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    keep = field((bi.double() + 0.5) * blk * h - 1.0).abs() <= band + 0.5 * math.sqrt(3.0) * blk * h
    ob = torch.arange(blk, device=DEV)
    off = torch.stack(torch.meshgrid(ob, ob, ob, indexing="ij"), -1).reshape(-1, 3)
    vox = (bi[keep][:, None] * blk + off[None]).reshape(-1, 3)
    vox = vox[(vox < res).all(1)]
    vox = vox[field((vox.double() + 0.5) * h - 1.0).abs() <= band]
    vox = vox[torch.argsort((vox[:, 0] * res + vox[:, 1]) * res + vox[:, 2])]
    corners = torch.tensor([[i & 1, (i >> 1) & 1, (i >> 2) & 1] for i in range(8)], device=DEV)
    p = res + 1
    c = vox[:, None] + corners[None]
    uv, inv = torch.unique((c[..., 0] * p + c[..., 1]) * p + c[..., 2], return_inverse=True)
    x = torch.stack([uv // (p * p), (uv // p) % p, uv % p], -1).double() * h - 1.0
    sdf = field(x) + 0.05 * h * torch.randn(x.shape[0], generator=g, dtype=F64, device=DEV)
    g = _gen(seed)
    sdf = sdf * (0.8 + 0.4 * torch.rand(x.shape[0], generator=g, dtype=F64, device=DEV))
    st = {"vox": vox.contiguous(), "sdf": sdf.float(), "cube": inv.reshape(-1, 8).contiguous(), "res": res}
    if case["weights"]:
        st["deform"] = (0.2 * h * (torch.rand(x.shape, generator=g, device=DEV) * 2 - 1)).float()
        st["alpha"] = 0.3 * torch.randn(vox.shape[0], 8, generator=g, device=DEV)
        st["beta"] = 0.3 * torch.randn(vox.shape[0], 12, generator=g, device=DEV)
    return st


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "query":
        v, f, p = _mesh_points(case, seed)
        st.update(mesh=MeshBVH(v, f), points=p, signed=case["signed"])
    elif kind == "adjoint":
        v, f, p = _mesh_points(case, seed)
        w = torch.randn(p.shape[0], generator=_gen(seed + 1), device=DEV)
        st.update(mesh=MeshBVH(v.requires_grad_(True), f), points=p.requires_grad_(True), weight=w)
    elif kind == "rebuild":
        v, f, p = _mesh_points(case, seed)
        st.update(vertices=v, faces=f, points=p)
    elif kind == "batch":
        meshes, p, counts = _batch_inputs(case, seed)
        st.update(batch=BatchedMeshBVH(meshes), points=p, counts=counts)
    elif kind == "rays":
        v, f, o, d = _mesh_rays(case, seed)
        st.update(mesh=MeshBVH(v, f), origins=o, directions=d)
    elif kind == "parity":
        v, f, p = _mesh_points(case, seed)
        st.update(mesh=MeshBVH(v, f), points=p, dirs=case["dirs"])
    elif kind in ("flood", "clip"):
        v, f = _voxel_mesh(case, seed)
        bounds = torch.tensor([[-1.0] * 3, [1.0] * 3], device=DEV)
        st.update(mesh=MeshBVH(v, f), bounds=bounds, level=case["level"],
                  octree=OctreeIndexer(max_level=case["level"], bounds=bounds, device=DEV),
                  connectivity=case.get("connectivity", 26))
    else:
        st.update(_dmc_inputs(case, seed), mode=case["mode"])
        st["module"] = SparseDiffDMC(device=DEV)
        if case["mode"] == "qef":
            st["module"].eval()
        else:
            for k in ("sdf", "deform", "alpha", "beta"):
                if k in st:
                    st[k].requires_grad_(True)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _min_level(level):
    return min(4, level - 1)


def run(state):
    kind = state["kind"]
    if kind == "query":
        call = state["mesh"].sdf if state["signed"] else state["mesh"].udf
        r = call(state["points"], return_closest=True, return_face_ids=True)
        return {"distances": r.distances, "closest": r.closest_points, "faces": r.face_ids}
    if kind == "adjoint":
        mesh, p = state["mesh"], state["points"]
        d = mesh.sdf(p, return_grad=True)
        gp, gv = torch.autograd.grad(d, [p, mesh.vertices], grad_outputs=state["weight"])
        return {"distances": d.detach(), "grad_points": gp, "grad_vertices": gv}
    if kind == "rebuild":
        mesh = MeshBVH(state["vertices"], state["faces"])
        r = mesh.udf(state["points"], return_closest=True)
        return {"distances": r.distances, "closest": r.closest_points, "face_normals": mesh.get_face_normals(),
                "vertex_normals": mesh.get_vertex_normals()}
    if kind == "batch":
        state["batch"].build()
        d, fid, cp = state["batch"].udf(state["points"], state["counts"])
        return {"distances": d, "closest": cp, "faces": fid}
    if kind == "rays":
        r = state["mesh"].intersect_ray(state["origins"], state["directions"], return_uvw=True)
        return {"hit": r.hit, "t": r.t, "faces": r.face_ids, "points": r.hit_points, "normals": r.normals,
                "bary": r.bary_coords}
    if kind == "parity":
        return {"distances": state["mesh"].sdf(state["points"], mode="parity", n_dirs=state["dirs"])}
    if kind == "flood":
        out = sparse_flood_fill(state["mesh"], 1 << state["level"], connectivity=state["connectivity"],
                                min_level=_min_level(state["level"]), bounds=state["bounds"], verbose=False)
        graph = construct_surface_dual_graph(out["dam_ijk"], out["tide_ijk"], out["dry_adjacent_ijk"],
                                             state["octree"])
        return {"labels": out, "graph": list(graph)}
    if kind == "clip":
        octree = state["octree"]
        cubes = octree.octree_traverse(state["mesh"], min_level=_min_level(state["level"]))
        lo, hi = octree.cube_aabb_level(cubes, state["level"])
        r = state["mesh"].intersect_aabb(lo, hi, mode=3)
        return {"cubes": cubes, "boxes": r.aabb_ids, "faces": r.face_ids, "centroids": r.centroids, "areas": r.areas,
                "polygons": r.poly_verts, "corners": r.poly_counts}
    o = state["module"](state["vox"], state["sdf"], state["cube"], state["res"], deform=state.get("deform"),
                        alpha=state.get("alpha"), beta=state.get("beta"))
    out = {"vertices": o.vertices.detach(), "faces": o.faces, "L_dev": o.L_dev.detach()}
    if state["mode"] == "train":
        leaves = [state[k] for k in ("sdf", "deform", "alpha", "beta") if k in state]
        loss = o.vertices.square().sum() + 0.1 * o.L_dev.sum()
        out["grads"] = list(torch.autograd.grad(loss, leaves))
    else:
        out["p_alpha"] = o.p_alpha
    return out


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once, and one evaluation of what
    each output is made of (the triangle of a closest point, a hit, a pair)."""
    kind = case["kind"]
    tri_b = 18.0  # 12 B of indices and half a 12-B vertex per triangle
    if kind in ("query", "adjoint", "rebuild", "parity"):
        n, t = case["points"], case["tris"]
        per = {"query": 32, "adjoint": 12 + 4 + 4 + 12, "rebuild": 12 + 4 + 12, "parity": 16}[kind]
        extra = {"adjoint": 6.0, "rebuild": 12 + 6.0}.get(kind, 0.0)
        return {"bytes": n * per + t * (tri_b + extra), "flops": n * 70.0 * (case["dirs"] if kind == "parity" else 1)}
    if kind == "rays":
        return {"bytes": case["rays"] * (24 + 1 + 4 + 4 + 12 + 12 + 12) + case["tris"] * tri_b,
                "flops": case["rays"] * 30.0}
    if kind == "batch":
        span = case["max_level"] - case["min_level"] + 1
        tris = sum(20 * 4 ** (case["min_level"] + i % span) for i in range(case["meshes"]))
        return {"bytes": tris * (tri_b + case["per_tri"] * 32.0), "flops": tris * case["per_tri"] * 70.0}
    if kind in ("flood", "clip"):
        cells = 4.0 * 4 ** case["level"]  # surface cells: about 2.8 R^2 for a ball of 0.9 of the box
        if kind == "clip":
            return {"bytes": cells * 24 + 1.7 * cells * (16 + 12 + 4 + 4 + 96) + case["tris"] * tri_b,
                    "flops": 1.7 * cells * 250.0}
        vox = 0.6 * 8.0 ** case["level"]  # labelled voxels, 12 B of coordinates each
        return {"bytes": vox * 12 + 2.5 * cells * (12 + 12 + 64 + 48 + 36) + case["tris"] * tri_b,
                "flops": cells * 130.0}
    # band of about 5 cells about spheres of mean radius 0.125 (overlaps left out)
    cubes = min(1.0, case["spheres"] / 40.0) * 40 * 4 * math.pi * 0.125 ** 2 * (case["res"] / 2.0) ** 2 * 4.7
    surf = cubes * 0.33
    per = 24 + 64 + 4 * 1.2 + ((12 * 1.2 + 32 + 48) if case["weights"] else 0)
    out = surf * (24 + 96 + 4 * 5)
    grads = cubes * (4 * 1.2 + ((12 * 1.2 + 32 + 48) if case["weights"] else 0)) if case["mode"] == "train" else 0
    return {"bytes": cubes * per + out + grads, "flops": surf * 4 * 60.0}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _closest(p, v, f):
    """Nearest face and closest point of each point by 64-bit brute force."""
    tri = v.double()[f.long()]
    a, ab, ac = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cab, cac = ab.T, ac.T
    d00, d01, d11 = (ab * ab).sum(1), (ab * ac).sum(1), (ac * ac).sum(1)
    bc = ac - ab
    dbc = (bc * bc).sum(1)
    den = d00 * d11 - d01 * d01
    pd = p.double()
    best = torch.empty(p.shape[0], dtype=torch.int64, device=DEV)
    step = max(1, (1 << 25) // max(1, f.shape[0]))
    for s in range(0, p.shape[0], step):
        q = pd[s:s + step]
        ap = [q[:, i:i + 1] - a[None, :, i] for i in range(3)]
        x, y, sq = _dot(ap, cab), _dot(ap, cac), _dot(ap, ap)
        v1, w1 = (d11 * x - d01 * y) / den, (d00 * y - d01 * x) / den
        inside = (v1 >= 0) & (w1 >= 0) & (v1 + w1 <= 1)
        dp = sq - v1 * x - w1 * y
        t = (x / d00).clamp(0, 1)
        d = sq - t * (2 * x - t * d00)
        t = (y / d11).clamp(0, 1)
        d = torch.minimum(d, sq - t * (2 * y - t * d11))
        # edge bc: p - b = ap - ab, (p - b).bc = (y - x) - ab.bc
        xb = (y - x) - (d01 - d00)
        sb = sq - 2 * x + d00
        t = (xb / dbc).clamp(0, 1)
        d = torch.minimum(d, sb - t * (2 * xb - t * dbc))
        best[s:s + step] = torch.where(inside, torch.minimum(d, dp), d).argmin(1)
    A, AB, AC = a[best], ab[best], ac[best]
    ap = pd - A
    x, y = (ap * AB).sum(1), (ap * AC).sum(1)
    v1 = (d11[best] * x - d01[best] * y) / den[best]
    w1 = (d00[best] * y - d01[best] * x) / den[best]
    cand = [(v1, w1)]
    t = (x / d00[best]).clamp(0, 1)
    cand.append((t, torch.zeros_like(t)))
    t = (y / d11[best]).clamp(0, 1)
    cand.append((torch.zeros_like(t), t))
    t = (((y - x) - (d01 - d00)[best]) / dbc[best]).clamp(0, 1)
    cand.append((1 - t, t))
    dist, bary, cp = None, None, None
    for k, (vv, ww) in enumerate(cand):
        c = A + vv[:, None] * AB + ww[:, None] * AC
        e = (pd - c).norm(dim=1)
        if k == 0:
            e = torch.where((vv >= 0) & (ww >= 0) & (vv + ww <= 1), e, torch.full_like(e, float("inf")))
            dist, bary, cp = e, torch.stack([1 - vv - ww, vv, ww], 1), c
        else:
            m = e < dist
            dist = torch.where(m, e, dist)
            bary = torch.where(m[:, None], torch.stack([1 - vv - ww, vv, ww], 1), bary)
            cp = torch.where(m[:, None], c, cp)
    return dist, best, bary, cp


def _normals(v, f):
    """Unit face normals and angle-weighted vertex normals."""
    fl = f.long()
    t = v.double()[fl]
    e = [t[:, (k + 1) % 3] - t[:, k] for k in range(3)]
    fn = torch.linalg.cross(e[0], -e[2])
    fn = fn / fn.norm(dim=1, keepdim=True)
    vn = torch.zeros(v.shape[0], 3, dtype=F64, device=DEV)
    for k in range(3):
        x, y = e[k], -e[(k + 2) % 3]
        ang = torch.atan2(torch.linalg.cross(x, y).norm(dim=1), (x * y).sum(1))
        vn.index_add_(0, fl[:, k], fn * ang[:, None])
    return fn, vn / vn.norm(dim=1, keepdim=True)


def _sign(p, v, f, face, bary, cp):
    """Pseudo-normal sign: face, edge or vertex normal of the closest feature."""
    fl = f.long()
    fn, vn = _normals(v, f)
    n = v.shape[0]
    a, b = fl, fl[:, [1, 2, 0]]
    key = (torch.minimum(a, b) * n + torch.maximum(a, b)).reshape(-1)
    uk, inv = torch.unique(key, return_inverse=True)
    en = torch.zeros(uk.shape[0], 3, dtype=F64, device=DEV).index_add_(0, inv, fn.repeat_interleave(3, 0))
    zero = bary < 1e-4
    nz = zero.sum(1)
    nrm = fn[face]
    # corner i opposite edge (i + 1, i + 2), which is half-edge i + 1 of the face
    half = (zero.int().argmax(1) + 1) % 3
    nrm = torch.where((nz == 1)[:, None], en[inv.reshape(-1, 3)[face, half]], nrm)
    nrm = torch.where((nz == 2)[:, None], vn[fl[face, bary.argmax(1)]], nrm)
    s = ((p.double() - cp) * nrm).sum(1)
    return torch.where(s < 0, -1.0, 1.0).double()


def _exact_rays(case, seed):
    v, f, o, d = _mesh_rays(case, seed)
    tri = v.double()[f.long()]
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    od, dd = o.double(), d.double()
    k = od.shape[0]
    t = torch.full((k,), float("inf"), dtype=F64, device=DEV)
    face = torch.zeros(k, dtype=torch.int64, device=DEV)
    step = max(1, (1 << 24) // f.shape[0])
    for s in range(0, k, step):
        D = [dd[s:s + step, i:i + 1] for i in range(3)]
        T = [od[s:s + step, i:i + 1] - a[None, :, i] for i in range(3)]
        cr = [T[1] * D[2] - T[2] * D[1], T[2] * D[0] - T[0] * D[2], T[0] * D[1] - T[1] * D[0]]  # T x D
        den = -_dot(D, n.T)
        u = -_dot(cr, e2.T) / den
        w = _dot(cr, e1.T) / den
        tt = _dot(T, n.T) / den
        tt = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (tt > 0), tt, torch.full_like(tt, float("inf")))
        t[s:s + step], face[s:s + step] = tt.min(1)
    hit = torch.isfinite(t)
    p = od + torch.where(hit, t, torch.zeros_like(t))[:, None] * dd
    fn = n / n.norm(dim=1, keepdim=True)
    return hit, t, p, fn[face]


def _linear_interp(w, x):
    """Zero crossing of two-point linear data w [.., 2, 1] at x [.., 2, C]."""
    return (x[..., 0, :] * w[..., 1, :] - x[..., 1, :] * w[..., 0, :]) / (w[..., 1, :] - w[..., 0, :])


def _exact_dmc(case, seed):
    st = _dmc_inputs(case, seed)
    res, vox, ci = st["res"], st["vox"], st["cube"]
    num_tab = torch.from_numpy(table("num_vd_table")).to(DEV)
    dmc_tab = torch.from_numpy(table("dmc_table")).to(DEV)
    chk_tab = torch.from_numpy(table("check_table")).to(DEV)
    edges = torch.tensor([0, 1, 1, 5, 4, 5, 0, 4, 2, 3, 3, 7, 6, 7, 2, 6, 2, 0, 3, 1, 7, 5, 6, 4], device=DEV)
    corners = torch.tensor([[i & 1, (i >> 1) & 1, (i >> 2) & 1] for i in range(8)], device=DEV)
    train = case["mode"] == "train"
    leaf = {k: st[k].double().requires_grad_(train) for k in ("sdf", "deform", "alpha", "beta") if k in st}
    s = leaf["sdf"]
    x = torch.zeros(s.shape[0], 3, dtype=F64, device=DEV)
    x[ci.reshape(-1)] = (vox[:, None] + corners).reshape(-1, 3).double() * (2.0 / res) - 1.0
    if "deform" in leaf:
        x = x + leaf["deform"]
    occ8 = (s.detach() < 0)[ci]
    surf = occ8.any(1) & ~occ8.all(1)
    if not bool(surf.any()):
        return None
    bits = (occ8[surf].long() << torch.arange(8, device=DEV)).sum(1)
    case_id = bits.clone()
    chk = chk_tab[bits]
    pc = vox[surf]
    adj = pc + chk[:, 1:4]
    ok = (chk[:, 0] == 1) & (adj >= 0).all(1) & (adj < res).all(1)
    # only the cubes whose own case is ambiguous are looked up
    amb = chk[:, 0] == 1
    hashes = torch.sort((pc[amb, 0] * res + pc[amb, 1]) * res + pc[amb, 2]).values
    if hashes.numel():
        ah = (adj[:, 0] * res + adj[:, 1]) * res + adj[:, 2]
        at = torch.searchsorted(hashes, ah).clamp(max=hashes.shape[0] - 1)
        ok &= hashes[at] == ah
        case_id = torch.where(ok, chk[:, 4], bits)
    cs = ci[surf]
    ones = torch.ones(surf.sum(), 1, dtype=F64, device=DEV)
    alpha = torch.tanh(leaf["alpha"][surf]) * 0.99 + 1 if "alpha" in leaf else ones.expand(-1, 8)
    beta = torch.tanh(leaf["beta"][surf]) * 0.99 + 1 if "beta" in leaf else ones.expand(-1, 12)
    num = num_tab[case_id]
    eg, vd, cube, total = [], [], [], 0
    for k in range(1, 5):
        cur = (num == k).nonzero()[:, 0]
        if cur.numel() == 0:
            continue
        tab = dmc_tab[case_id[cur], :k].reshape(-1, 7)
        row = torch.arange(tab.shape[0], device=DEV)[:, None].expand(-1, 7) + total
        m = tab != -1
        eg.append(tab[m])
        vd.append(row[m])
        cube.append(cur.repeat_interleave(k)[:, None].expand(-1, 7)[m])
        total += tab.shape[0]
    eg, vd, cube = torch.cat(eg), torch.cat(vd), torch.cat(cube)
    ends = cs[:, edges].reshape(-1, 12, 2)[cube, eg]
    xs, ss = x[ends], s[ends][..., None]
    zc = _linear_interp(ss, xs)
    ue = _linear_interp(ss * alpha[:, edges].reshape(-1, 12, 2)[cube, eg][..., None], xs)
    b = beta[cube, eg][:, None]
    cnt = torch.zeros(total, dtype=F64, device=DEV).index_add_(0, vd, torch.ones_like(vd, dtype=F64))

    def fold(val):
        return torch.zeros(total, val.shape[1], dtype=F64, device=DEV).index_add(0, vd, val)

    def l_dev(pos):
        d = (zc - pos[vd]).norm(dim=1)
        return (d - (fold(d[:, None])[:, 0] / cnt)[vd]).abs()

    if not train:
        return {"vertices": None, "faces": None, "L_dev": None, "p_alpha": ue.detach()}
    pos = fold(ue * b) / fold(b)
    ld = l_dev(pos)
    # quads: the crossing edges that four active cubes share, in edge order
    all_e = cs[:, edges].reshape(-1, 2)
    uk, inv, count = torch.unique(all_e[:, 0] * s.shape[0] + all_e[:, 1], return_inverse=True, return_counts=True)
    o = s.detach() < 0
    cross = (o[all_e[:, 0]] != o[all_e[:, 1]]) & (count[inv] == 4)
    slot = torch.zeros(all_e.shape[0], dtype=torch.int64, device=DEV)
    slot[cube * 12 + eg] = vd
    order = torch.argsort(inv[cross], stable=True)
    quad = slot[cross][order].reshape(-1, 4)
    verts = torch.cat([pos, pos[quad].mean(1)])
    loss = verts.square().sum() + 0.1 * ld.sum()
    keys = [k for k in ("sdf", "deform", "alpha", "beta") if k in leaf]
    grads = torch.autograd.grad(loss, [leaf[k] for k in keys])
    return {"vertices": verts.detach(), "faces": None, "L_dev": ld.detach(), "grads": list(grads)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("query", "adjoint", "rebuild", "parity"):
        if float(case["points"]) * case["tris"] > EXACT_PAIRS:
            return None
        v, f, p = _mesh_points(case, seed)
        d, face, bary, cp = _closest(p, v, f)
        if kind == "parity":
            return {"distances": d * _sign(p, v, f, face, bary, cp)}
        if kind == "rebuild":
            fn, vn = _normals(v, f)
            return {"distances": d, "closest": cp, "face_normals": fn, "vertex_normals": vn}
        if kind == "query":
            if case["signed"]:
                d = d * _sign(p, v, f, face, bary, cp)
            return {"distances": d, "closest": cp, "faces": None}
        w = torch.randn(p.shape[0], generator=_gen(seed + 1), device=DEV).double()
        s = _sign(p, v, f, face, bary, cp)
        gp = (w * s / d)[:, None] * (p.double() - cp)
        gv = torch.zeros(v.shape[0], 3, dtype=F64, device=DEV)
        for k in range(3):
            gv.index_add_(0, f[face, k].long(), -bary[:, k:k + 1] * gp)
        return {"distances": d * s, "grad_points": gp, "grad_vertices": gv}
    if kind == "rays":
        if float(case["rays"]) * case["tris"] > EXACT_PAIRS:
            return None
        hit, t, p, n = _exact_rays(case, seed)
        return {"hit": None, "t": t, "faces": None, "points": None, "normals": None, "bary": None}
    if kind == "batch":
        tris = sum(20 * 4 ** (case["min_level"] + i % (case["max_level"] - case["min_level"] + 1))
                   for i in range(case["meshes"]))
        if case["per_tri"] * (20.0 * 4 ** case["max_level"]) * tris > EXACT_PAIRS:
            return None
        meshes, p, counts = _batch_inputs(case, seed)
        parts, at = [], 0
        for (v, f), n in zip(meshes, counts):
            parts.append(_closest(p[at:at + n], v, f))
            at += n
        return {"distances": torch.cat([x[0] for x in parts]), "closest": torch.cat([x[3] for x in parts]),
                "faces": None}
    if kind == "dmc":
        return _exact_dmc(case, seed)
    return None  # voxel labels, indices and clip polygons in the tree's own order
