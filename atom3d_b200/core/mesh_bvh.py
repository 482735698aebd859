"""MeshBVH: the mesh query object (drop-in for atom3d.core.mesh_bvh.MeshBVH).

Keeps the reference's constructor and query signatures
(atom3d/core/mesh_bvh.py:59-117, :297-335, :601-757) while every
computation runs in libatom3d_b200.so on the GPU:

* construction: pseudo-normal precompute (a3d_mesh_normals) and the GPU
  wide-BVH build (a3d_bvh_build_children) instead of the reference's host SAH
  build;
* ``udf`` / ``sdf``: one native call (a3d_udf_children), traversal and outputs,
  sign included;
* ``udf(return_grad=True)``: a torch.autograd.Function whose backward is the
  hand-written adjoint kernel (a3d_udf_backward) for points and vertices;
* ``intersect_aabb``: SAT any-hit over the BVH (mode 0, a3d_aabb_hit) and
  the (box, face) pairs, clipped for modes 2-3 (a3d_aabb_pairs_*).

There is no CPU path: a CPU device raises.
"""

from __future__ import annotations

import ctypes
import os
from typing import Optional, Union

import torch

from .. import _lib
from .data_structures import AABBIntersectResult, ClosestPointResult, RayAllHitResult, RayIntersectResult
from .device_utils import resolve_device


class WideBVH:
    """Device-resident 4-wide quantised BVH (64-B nodes, 64-B triangle records)."""

    DEFAULT_LEAF_MAX = int(os.environ.get("ATOM3D_B200_LEAF_MAX", "8"))

    def __init__(self, vertices: torch.Tensor, faces: torch.Tensor, leaf_max: int | None = None):
        _lib.require_cuda(vertices, "vertices")
        self.leaf_max = int(leaf_max or self.DEFAULT_LEAF_MAX)
        dev = vertices.device
        v = vertices.detach().contiguous().float()
        f = faces.contiguous().int()
        nf = int(f.shape[0])
        if nf == 0:
            raise ValueError("MeshBVH needs at least one face")
        self.device = dev
        self.num_tris = nf
        cap = max(nf, 1)
        with torch.cuda.device(dev):
            nodes = torch.empty(cap * 64 + 64, dtype=torch.uint8, device=dev)
            off = (-nodes.data_ptr()) % 64
            nodes = nodes[off:off + cap * 64]
            tris = torch.empty(nf * 64, dtype=torch.uint8, device=dev)
            ws = _lib.workspace(_lib.lib().a3d_bvh_build_workspace_bytes(nf), dev)
            nn = ctypes.c_int64(0)
            bounds = (ctypes.c_float * 6)()
            # child records: decoded boxes and discs for the closest-point traversal
            ccap = self._child_capacity(nf, self.leaf_max)
            children = self._child_buffer(ccap, nf, dev)
            _lib.call(
                "a3d_bvh_build_children", v.data_ptr(), v.shape[0], f.data_ptr(), nf, self.leaf_max, nodes.data_ptr(),
                cap, tris.data_ptr(), children.data_ptr(), ccap, ws.data_ptr(), ws.numel(), ctypes.byref(nn), bounds,
                _lib.stream_ptr(dev),
            )
            self.num_nodes = int(nn.value)
            if self.num_nodes > ccap:
                children = self._child_buffer(self.num_nodes, nf, dev)
                _lib.call("a3d_bvh_children", nodes.data_ptr(), tris.data_ptr(), self.num_nodes, None, nf,
                          children.data_ptr(), _lib.stream_ptr(dev))
                torch.cuda.current_stream(dev).synchronize()
            self.nodes = nodes[: self.num_nodes * 64]
            self.tris = tris
            self.children = children
        self.lo = [bounds[0], bounds[1], bounds[2]]
        self.hi = [bounds[3], bounds[4], bounds[5]]
        self._view = _lib.BvhView(
            self.nodes.data_ptr(), self.tris.data_ptr(), self.num_nodes, self.num_tris,
            (ctypes.c_float * 3)(*self.lo), (ctypes.c_float * 3)(*self.hi),
        )

    @staticmethod
    def _child_capacity(nf: int, leaf_max: int) -> int:
        """Nodes to hold child records for, before the tree is known: leaves of
        up to 8 triangles make about nf / 12 nodes, of one triangle nf / 3."""
        return nf // (8 if leaf_max >= 8 else 2) + 64

    @staticmethod
    def _child_buffer(nodes: int, nf: int, dev) -> torch.Tensor:
        return torch.empty(_lib.lib().a3d_bvh_children_bytes(nodes, nf), dtype=torch.uint8, device=dev)

    @property
    def view(self) -> _lib.BvhView:
        return self._view

    def query(self, points: torch.Tensor, sign: Optional[_lib.SignData] = None, bound: Optional[torch.Tensor] = None,
              want_uvw: bool = True, stats: Optional[torch.Tensor] = None, sort_queries: bool = True,
              seeding: int = 0):
        """Raw closest-point query: (distances, face_ids int32, closest [N,3], uvw [N,3] or None)."""
        _lib.require_cuda(points, "points")
        p = points.detach().contiguous().float()
        n = int(p.shape[0])
        dev = self.device
        dist = torch.empty(n, dtype=torch.float32, device=dev)
        fid = torch.empty(n, dtype=torch.int32, device=dev)
        cp = torch.empty(n, 3, dtype=torch.float32, device=dev)
        uvw = torch.empty(n, 3, dtype=torch.float32, device=dev) if want_uvw else None
        if n == 0:
            return dist, fid, cp, uvw
        flags = (_lib.A3D_UDF_SORT_QUERIES if sort_queries else 0) | seeding
        ws = _lib.workspace(_lib.lib().a3d_udf_workspace_bytes(n, flags), dev)
        self._last_ws = ws
        b = None
        if bound is not None:
            b = bound.detach().contiguous().float()
            if b.shape[0] != n:
                raise ValueError("bound must have one entry per query")
        _lib.call(
            "a3d_udf_children", ctypes.byref(self._view), self.children.data_ptr(), p.data_ptr(), n, dist.data_ptr(),
            fid.data_ptr(), cp.data_ptr(), _lib.ptr(uvw), ctypes.byref(sign) if sign is not None else None,
            _lib.ptr(b), _lib.ptr(stats), flags, ws.data_ptr(), ws.numel(), _lib.stream_ptr(dev),
        )
        return dist, fid, cp, uvw


    def status(self) -> dict:
        """Status words of the last query (synchronises): queries re-run,
        deep-stack overflow, guard faults."""
        return udf_status(self._last_ws, self.device)


def udf_status(ws: torch.Tensor, device) -> dict:
    """Read the status words a query left at the start of its workspace."""
    st = (ctypes.c_uint32 * 4)()
    _lib.call("a3d_udf_status", ws.data_ptr(), st, _lib.stream_ptr(device))
    return {"reruns": int(st[0]), "overflow": int(st[1]), "faults": int(st[3])}


class _DistanceFn(torch.autograd.Function):
    """dist(points, vertices) with the hand-written adjoint kernel.

    Forward runs the (optionally signed) closest-point query; backward calls
    a3d_udf_backward: d|p-c|/dp = (p-c)/|p-c| and, by the envelope theorem,
    d|p-c|/dv_i = -w_i (p-c)/|p-c| with w the closest point's barycentrics.
    """

    @staticmethod
    def forward(ctx, points, vertices, mesh, sign_flag, bound):
        dist, fid, cp, uvw = mesh._bvh.query(points, sign=mesh._sign_data() if sign_flag else None, bound=bound)
        ctx.mesh = mesh
        ctx.save_for_backward(points, cp, fid, uvw, dist)
        ctx.mark_non_differentiable(fid, cp, uvw)
        return dist, fid, cp, uvw

    @staticmethod
    def backward(ctx, g_dist, _g_fid, _g_cp, _g_uvw):
        points, cp, fid, uvw, dist = ctx.saved_tensors
        mesh = ctx.mesh
        need_p, need_v = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
        if g_dist is None or not (need_p or need_v):
            return None, None, None, None, None
        # signed distance = sign * |p - c|: fold the sign into the incoming grad
        g = (g_dist * torch.where(dist < 0, -1.0, 1.0)).contiguous().float()
        n = points.shape[0]
        gp = torch.empty(n, 3, dtype=torch.float32, device=points.device) if need_p else None
        gv = torch.zeros_like(mesh.vertices, dtype=torch.float32) if need_v else None
        _lib.call(
            "a3d_udf_backward", points.detach().contiguous().float().data_ptr(), n, cp.data_ptr(), fid.data_ptr(),
            uvw.data_ptr(), g.data_ptr(), mesh.faces.data_ptr(), _lib.ptr(gp), _lib.ptr(gv),
            _lib.stream_ptr(points.device),
        )
        if gp is not None:
            gp = gp.to(points.dtype)
        return gp, gv, None, None, None


class MeshBVH:
    """Mesh with a GPU wide BVH; closest-point, signed-distance and box queries.

    Args:
        vertices: [V, 3] vertex coordinates
        faces: [F, 3] vertex indices
        device: compute device (must resolve to CUDA)
        face_normals: optional [F, 3] normals used by the sign test
        vertex_normals: optional [V, 3] vertex normals (then the sign uses
            face normals only, like the reference)
    """

    def __init__(
        self,
        vertices: torch.Tensor,
        faces: torch.Tensor,
        device: Optional[Union[str, torch.device]] = None,
        face_normals: Optional[torch.Tensor] = None,
        vertex_normals: Optional[torch.Tensor] = None,
    ):
        dev = resolve_device(vertices, faces, device=device, default="cuda")
        if dev.type != "cuda":
            raise RuntimeError(
                f"MeshBVH runs on CUDA only (resolved device {dev}); there is no CPU fallback"
            )
        if dev.index is None:
            dev = torch.device("cuda", torch.cuda.current_device())
        self.device = dev
        self.vertices = vertices.to(dev).float()
        self.faces = faces.to(dev).int().contiguous()
        self.num_vertices = int(self.vertices.shape[0])
        self.num_faces = int(self.faces.shape[0])
        vd = self.vertices.detach()
        self._bounds = torch.stack([vd.min(dim=0)[0], vd.max(dim=0)[0]])
        self._is_cuda = True
        self._edge_pn = None
        self._he_edge_idx = None
        self._face_angles = None
        self._precompute_normals()
        if face_normals is not None:
            self._face_normals = face_normals.to(dev).float().contiguous()
        if vertex_normals is not None:
            self._vertex_pn = vertex_normals.to(dev).float().contiguous()
            self._edge_pn = None
            self._he_edge_idx = None
            self._face_angles = None
        self._vertex_normals = self._vertex_pn
        self._bvh = WideBVH(vd, self.faces)
        self._sign_cache = None

    # ------------------------------------------------------------------ setup
    def _precompute_normals(self) -> None:
        dev = self.device
        nv, nf = self.num_vertices, self.num_faces
        v = self.vertices.detach().contiguous()
        fn = torch.empty(nf, 3, dtype=torch.float32, device=dev)
        ang = torch.empty(nf, 3, dtype=torch.float32, device=dev)
        vpn = torch.empty(nv, 3, dtype=torch.float32, device=dev)
        epn = torch.empty(3 * nf, 3, dtype=torch.float32, device=dev)
        he = torch.empty(3 * nf, dtype=torch.int64, device=dev)
        ne = ctypes.c_int64(0)
        ws = _lib.workspace(_lib.lib().a3d_mesh_normals_workspace_bytes(nv, nf), dev)
        _lib.call(
            "a3d_mesh_normals", v.data_ptr(), nv, self.faces.data_ptr(), nf, fn.data_ptr(), ang.data_ptr(),
            vpn.data_ptr(), epn.data_ptr(), 3 * nf, he.data_ptr(), ctypes.byref(ne), ws.data_ptr(), ws.numel(),
            _lib.stream_ptr(dev),
        )
        self._face_normals = fn
        self._face_angles = ang
        self._vertex_pn = vpn
        self._edge_pn = epn[: int(ne.value)]
        self._he_edge_idx = he

    def _sign_data(self) -> _lib.SignData:
        key = (id(self._face_normals), id(self._vertex_pn), id(self._edge_pn))
        if self._sign_cache is None or self._sign_cache[0] != key:
            face_only = self._edge_pn is None or self._he_edge_idx is None
            sd = _lib.SignData(
                self._face_normals.data_ptr(),
                None if face_only else self._vertex_pn.data_ptr(),
                None if face_only else self._edge_pn.data_ptr(),
                None if face_only else self._he_edge_idx.data_ptr(),
                self.faces.data_ptr(),
            )
            self._sign_cache = (key, sd)
        return self._sign_cache[1]

    # ------------------------------------------------------------- properties
    def get_bounds(self) -> torch.Tensor:
        return self._bounds

    def get_face_normals(self) -> torch.Tensor:
        return self._face_normals

    def get_vertex_normals(self) -> Optional[torch.Tensor]:
        return self._vertex_normals

    def get_face_aabb(self, face_indices: Optional[torch.Tensor] = None):
        f = self.faces if face_indices is None else self.faces[face_indices]
        tv = self.vertices.detach()[f.long()]
        return tv.min(dim=1)[0], tv.max(dim=1)[0]

    # ------------------------------------------------------------ box queries
    def intersect_aabb(self, aabb_min: torch.Tensor, aabb_max: torch.Tensor, mode: int = 1) -> AABBIntersectResult:
        """Triangle/box intersection (atom3d/core/mesh_bvh.py:297-479).

        mode 0: hit mask (some face passes SAT, sat_eps 1e-6)
        mode 1: hit mask + (aabb_ids, face_ids) int32 pairs passing SAT
        mode 2: pairs whose Sutherland-Hodgman clip against the box is
                non-empty (int64 ids), with centroids [P,3] (polygon mean
                clamped to the box, projected onto the triangle), areas [P]
                and poly_counts [P] int32; hit = box has such a pair
        mode 3: mode 2 plus poly_verts [P,8,3] (zero padded)
        Pairs come grouped by box in ascending order (tree order within a
        box); the reference returns them in atomic-counter order.
        """
        if mode == 0:
            return AABBIntersectResult(hit=self.aabb_hit(aabb_min, aabb_max))
        if mode not in (1, 2, 3):
            raise ValueError(f"intersect_aabb: mode must be 0, 1, 2 or 3, got {mode}")
        _lib.require_cuda(aabb_min, "aabb_min")
        mn = aabb_min.detach().contiguous().float()
        mx = aabb_max.detach().contiguous().float()
        n = int(mn.shape[0])
        dev = self.device
        hit = torch.zeros(n, dtype=torch.bool, device=dev)
        idt = torch.int32 if mode == 1 else torch.int64
        if n == 0:
            e = torch.empty(0, dtype=idt, device=dev)
            return AABBIntersectResult(hit=hit, aabb_ids=e, face_ids=e.clone()) if mode == 1 else \
                AABBIntersectResult(hit=hit)
        lib = _lib.lib()
        ws = _lib.workspace(lib.a3d_aabb_pairs_workspace_bytes(n), dev)
        stream = _lib.stream_ptr(dev)
        n_cand = ctypes.c_int64(0)
        _lib.call("a3d_aabb_pairs_count", ctypes.byref(self._bvh.view), mn.data_ptr(), mx.data_ptr(), n, mode,
                  hit.data_ptr(), ws.data_ptr(), ws.numel(), ctypes.byref(n_cand), stream)
        m = int(n_cand.value)
        if mode >= 2 and m == 0:
            return AABBIntersectResult(hit=hit)  # no SAT candidate at all: the reference returns the mask alone
        cws = None
        P = m
        if mode >= 2:
            cws = _lib.workspace(lib.a3d_aabb_clip_workspace_bytes(m), dev)
            n_pairs = ctypes.c_int64(0)
            _lib.call("a3d_aabb_pairs_clip", ctypes.byref(self._bvh.view), mn.data_ptr(), mx.data_ptr(), n,
                      ws.data_ptr(), ws.numel(), cws.data_ptr(), cws.numel(), m, hit.data_ptr(), ctypes.byref(n_pairs),
                      stream)
            P = int(n_pairs.value)
        a_ids = torch.empty(P, dtype=idt, device=dev)
        f_ids = torch.empty(P, dtype=idt, device=dev)
        pc = cen = ar = pv = None
        if mode >= 2:
            pc = torch.empty(P, dtype=torch.int32, device=dev)
            cen = torch.empty(P, 3, dtype=torch.float32, device=dev)
            ar = torch.empty(P, dtype=torch.float32, device=dev)
        if mode == 3:
            pv = torch.empty(P, 8, 3, dtype=torch.float32, device=dev)
        if P:
            ptr = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
            _lib.call("a3d_aabb_pairs_write", ctypes.byref(self._bvh.view), mn.data_ptr(), mx.data_ptr(), n, mode,
                      ws.data_ptr(), ws.numel(), ptr(cws), cws.numel() if cws is not None else 0, m,
                      a_ids.data_ptr(), f_ids.data_ptr(), ptr(pc), ptr(cen), ptr(ar), ptr(pv), stream)
        return AABBIntersectResult(hit=hit, aabb_ids=a_ids, face_ids=f_ids, centroids=cen, areas=ar, poly_verts=pv,
                                   poly_counts=pc)

    def aabb_hit(self, aabb_min: torch.Tensor, aabb_max: torch.Tensor) -> torch.Tensor:
        _lib.require_cuda(aabb_min, "aabb_min")
        mn = aabb_min.detach().contiguous().float()
        mx = aabb_max.detach().contiguous().float()
        n = int(mn.shape[0])
        hit = torch.zeros(n, dtype=torch.bool, device=self.device)
        if n == 0:
            return hit
        ws = _lib.workspace(_lib.lib().a3d_aabb_hit_workspace_bytes(n), self.device)
        _lib.call(
            "a3d_aabb_hit", ctypes.byref(self._bvh.view), mn.data_ptr(), mx.data_ptr(), n, hit.data_ptr(),
            ws.data_ptr(), ws.numel(), _lib.stream_ptr(self.device),
        )
        return hit

    # -------------------------------------------------------- distance queries
    def udf(
        self,
        points: torch.Tensor,
        return_grad: bool = False,
        return_closest: bool = False,
        return_uvw: bool = False,
        return_face_ids: bool = False,
        bound: Optional[torch.Tensor] = None,
    ) -> Union[torch.Tensor, ClosestPointResult]:
        """Unsigned distance (reference: atom3d/core/mesh_bvh.py:601-648).

        ``bound`` (extension): per-query upper bound on the distance used to
        seed the pruning radius; results are identical with or without it.
        """
        result = self._udf_with_grad(points, bound=bound) if return_grad else self._udf_query(points, bound=bound)
        return self._filter(result, return_closest, return_uvw, return_face_ids)

    def sdf(
        self,
        points: torch.Tensor,
        mode: str = "pseudo_normal",
        return_grad: bool = False,
        return_closest: bool = False,
        return_uvw: bool = False,
        return_face_ids: bool = False,
        bound: Optional[torch.Tensor] = None,
        **kwargs,
    ) -> Union[torch.Tensor, ClosestPointResult]:
        """Signed distance with the Baerentzen-Aanaes pseudo-normal sign
        (reference: atom3d/core/mesh_bvh.py:702-827), fused into the query."""
        if mode == "parity":
            return self._sdf_parity(points, **kwargs)
        if mode != "pseudo_normal":
            raise ValueError(f"sdf mode {mode!r}: use 'pseudo_normal' or 'parity'")
        if return_grad:
            result = self._udf_with_grad(points, sign=True, bound=bound)
        else:
            result = self._udf_query(points, sign=True, bound=bound)
        return self._filter(result, return_closest, return_uvw, return_face_ids)

    # ---------------------------------------------------------------- rays
    def intersect_ray(self, rays_o: torch.Tensor, rays_d: torch.Tensor, max_t: float = 1e10,
                      return_uvw: bool = False, mode: str = "nearest"):
        """Ray-mesh intersection (reference: atom3d/core/mesh_bvh.py:1076-1160).

        mode "nearest": closest hit per ray (RayIntersectResult); "all": every
        non-grazing hit, grouped by ray (RayAllHitResult).
        """
        if mode == "all":
            return self._intersect_ray_all(rays_o, rays_d, max_t)
        if mode != "nearest":
            raise ValueError(f"intersect_ray mode {mode!r}: use 'nearest' or 'all'")
        o, d = self._rays(rays_o, rays_d)
        n = o.shape[0]
        dev = self.device
        hit = torch.empty(n, dtype=torch.bool, device=dev)
        t = torch.empty(n, dtype=torch.float32, device=dev)
        fid = torch.empty(n, dtype=torch.int32, device=dev)
        hp = torch.empty(n, 3, dtype=torch.float32, device=dev)
        nrm = torch.empty(n, 3, dtype=torch.float32, device=dev)
        uvw = torch.empty(n, 3, dtype=torch.float32, device=dev) if return_uvw else None
        ws = _lib.workspace(_lib.lib().a3d_ray_workspace_bytes(n), dev)
        self._last_ray_ws = ws
        _lib.call("a3d_ray_nearest", ctypes.byref(self._bvh.view), o.data_ptr(), d.data_ptr(), n, float(max_t),
                  self._face_normals.data_ptr(), hit.data_ptr(), t.data_ptr(), fid.data_ptr(), hp.data_ptr(),
                  nrm.data_ptr(), _lib.ptr(uvw), ws.data_ptr(), ws.numel(), _lib.stream_ptr(dev))
        return RayIntersectResult(hit=hit, t=t, face_ids=fid, hit_points=hp, normals=nrm, bary_coords=uvw)

    def _rays(self, rays_o: torch.Tensor, rays_d: torch.Tensor):
        _lib.require_cuda(rays_o, "rays_o")
        _lib.require_cuda(rays_d, "rays_d")
        o = rays_o.detach().to(self.device).float().contiguous()
        d = rays_d.detach().to(self.device).float().contiguous()
        if o.shape != d.shape or o.dim() != 2 or o.shape[1] != 3:
            raise ValueError("rays_o and rays_d must both be [N, 3]")
        return o, d

    def _intersect_ray_all(self, rays_o: torch.Tensor, rays_d: torch.Tensor, max_t: float = 1e10) -> RayAllHitResult:
        o, d = self._rays(rays_o, rays_d)
        n = o.shape[0]
        dev = self.device
        lib = _lib.lib()
        ws = _lib.workspace(lib.a3d_ray_workspace_bytes(n), dev)
        self._last_ray_ws = ws
        offs = torch.empty(n + 1, dtype=torch.int64, device=dev)
        st = _lib.stream_ptr(dev)
        _lib.call("a3d_ray_all_count", ctypes.byref(self._bvh.view), o.data_ptr(), d.data_ptr(), n, float(max_t),
                  offs.data_ptr(), ws.data_ptr(), ws.numel(), st)
        total = int(offs[n].item()) if n else 0
        ray_idx = torch.empty(total, dtype=torch.int32, device=dev)
        t = torch.empty(total, dtype=torch.float32, device=dev)
        fid = torch.empty(total, dtype=torch.int32, device=dev)
        sign = torch.empty(total, dtype=torch.int32, device=dev)
        hp = torch.empty(total, 3, dtype=torch.float32, device=dev)
        uvw = torch.empty(total, 3, dtype=torch.float32, device=dev)
        if total:
            _lib.call("a3d_ray_all_collect", ctypes.byref(self._bvh.view), o.data_ptr(), d.data_ptr(), n,
                      float(max_t), offs.data_ptr(), ray_idx.data_ptr(), t.data_ptr(), fid.data_ptr(),
                      sign.data_ptr(), hp.data_ptr(), uvw.data_ptr(), st)
        return RayAllHitResult(ray_idx=ray_idx, t=t, face_ids=fid, sign=sign, hit_points=hp, bary_coords=uvw)

    def ray_status(self) -> dict:
        """Status of the last ray call (synchronises): rays re-run with the
        deep stack, and whether a stack or hit buffer overflowed."""
        st = (ctypes.c_uint32 * 2)()
        _lib.call("a3d_ray_status", self._last_ray_ws.data_ptr(), st, _lib.stream_ptr(self.device))
        return {"reruns": int(st[0]), "overflow": int(st[1])}

    def _sdf_parity(self, points: torch.Tensor, n_dirs: int = 8, max_t: float = 1e6, coalesce_t: float = 1e-4,
                    seed: int = 42, **_unused) -> torch.Tensor:
        """Signed distance with the ray-parity sign (reference:
        atom3d/core/mesh_bvh.py:850-948): for n_dirs seeded random
        directions, hits within coalesce_t along a ray are merged and the
        signed crossing count taken; a point is inside when more than half of
        the directions give an odd count.  All directions are traced by one
        fused kernel (traverse, sort by t, merge, vote)."""
        _lib.require_cuda(points, "points")
        p = points.detach().to(self.device).float().contiguous()
        n = p.shape[0]
        udf = self.udf(p)
        gen = torch.Generator(device=self.device)
        gen.manual_seed(seed)
        dirs = torch.randn(n_dirs, 3, device=self.device, generator=gen)
        dirs = (dirs / dirs.norm(dim=1, keepdim=True)).contiguous()
        votes = torch.empty(n, dtype=torch.int32, device=self.device)
        ws = _lib.workspace(_lib.lib().a3d_ray_workspace_bytes(0), self.device)
        self._last_ray_ws = ws
        _lib.call("a3d_ray_parity_votes", ctypes.byref(self._bvh.view), p.data_ptr(), n, dirs.data_ptr(), int(n_dirs),
                  float(max_t), float(coalesce_t), votes.data_ptr(), ws.data_ptr(), ws.numel(),
                  _lib.stream_ptr(self.device))
        inside = votes > (n_dirs // 2)
        return torch.where(inside, -udf, udf)

    @staticmethod
    def _filter(result: ClosestPointResult, closest: bool, uvw: bool, fids: bool):
        if not (closest or uvw or fids):
            return result.distances
        if not closest:
            result.closest_points = None
        if not uvw:
            result.uvw = None
        if not fids:
            result.face_ids = None
        return result

    def _udf_query(self, points: torch.Tensor, sign: bool = False, bound: Optional[torch.Tensor] = None):
        dist, fid, cp, uvw = self._bvh.query(points, sign=self._sign_data() if sign else None, bound=bound)
        return ClosestPointResult(distances=dist, face_ids=fid, closest_points=cp, uvw=uvw)

    def _udf_with_grad(self, points: torch.Tensor, sign: bool = False, bound: Optional[torch.Tensor] = None):
        dist, fid, cp, uvw = _DistanceFn.apply(points, self.vertices, self, sign, bound)
        return ClosestPointResult(distances=dist, face_ids=fid, closest_points=cp.detach(), uvw=uvw)

    def _compute_sign(self, points: torch.Tensor, closest_points=None, face_ids=None, uvw=None) -> torch.Tensor:
        """Sign (+1/-1) of the signed distance at ``points`` (fused kernel)."""
        d = self._udf_query(points, sign=True).distances
        return torch.where(d < 0, -1.0, 1.0)
