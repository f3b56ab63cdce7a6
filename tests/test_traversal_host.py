"""The device traversal run on the host (traversal_host.cpp): rays shared among a warp's lanes.

Unset lane state holds a pattern and reads outside the scene's arrays are counted, so these tests
see on the CPU what a helper lane that never loaded a ray of its own works with. Hits at the
ray's origin (t = +0 or -0) follow the tie rule here and on the GPU.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import binding as O


def _build(tmp, defines=()):
    from merian_gb300 import build as B
    lib = tmp / "libtraversal.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ftrivial-auto-var-init=pattern",
                    "-ffp-contract=off", "-fPIC", "-shared", *[f"-D{d}" for d in defines],
                    "-I", str(B.INCLUDE), "-I", str(B.CSRC), "-I",
                    str(B._cuda_home() / "include"), str(ROOT / "tests" / "traversal_host.cpp"),
                    "-o", str(lib)], check=True)
    fn = C.CDLL(str(lib)).traversal_host
    fn.restype = C.c_int64
    vp, u32, u64, i32 = C.c_void_p, C.c_uint32, C.c_uint64, C.c_int
    fn.argtypes = [vp, u64, vp, u64, vp, u64, i32, i32, vp, vp, u32, u32, u32, vp]
    return fn


@pytest.fixture(scope="module")
def host(native, tmp_path_factory):
    return _build(tmp_path_factory.mktemp("traversal"))


def _soup():
    from merian_gb300 import scene as S
    return S.soup(n_triangles=4000, n_geometries=8, env_size=None)


def _instances(sc, axes):
    """Eight overlapping instances of one BLAS: translations by sixteenths and, with `axes`, a
    permutation of the axes; their inverses are exact."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    rng = np.random.default_rng(4)
    inst = np.zeros(8, N.INSTANCE_DTYPE)
    for k in range(8):
        m = np.zeros((3, 4), np.float32)
        m[:, :3] = np.roll(np.eye(3), k if axes else 0, axis=0)
        m[:, 3] = np.round(rng.uniform(0, 0.75, 3) * 16) / 16
        inst["object_to_world"][k] = m.reshape(inst["object_to_world"][k].shape)
        inst["blas"][k] = 0
        inst["mask"][k] = 0xFF
    blas = np.zeros(1, N.BLAS_DTYPE)
    blas["first_geometry"] = 0
    blas["geometry_count"] = len(sc.geometries)
    return S.SceneData(sc.vertices, sc.indices, sc.geometries, sc.materials, None,
                       blas_ranges=blas, instances=inst)


def _records(sc, nodes, blas_nodes):
    """The upload's instance records: both transforms, BLAS root node, mask, first geometry."""
    rec = np.zeros((len(sc.instances), 28), np.float32)
    for k, i in enumerate(sc.instances):
        m = np.asarray(i["object_to_world"], np.float64).reshape(3, 4)
        rec[k, :12] = m.reshape(-1)
        inv = m[:, :3].T
        rec[k, 12:24] = np.concatenate([inv, -(inv @ m[:, 3:])], 1).reshape(-1)
        rec[k, 24:].view(np.uint32)[:] = [len(nodes) - blas_nodes, int(i["mask"]), 0, 0]
    return rec


def _run(host, nodes, tris, insts, rays, any_hit, mixed, per_ray, grid):
    from merian_gb300 import _native as N
    hits = np.zeros(len(rays), N.HIT_DTYPE)
    any_hit = np.ascontiguousarray(any_hit, np.uint8)
    bad = host(nodes.ctypes.data, len(nodes), tris.ctypes.data, len(tris),
               insts.ctypes.data if insts is not None else None,
               0 if insts is None else len(insts), mixed, per_ray, rays.ctypes.data,
               any_hit.ctypes.data, len(rays), 0xFF, grid, hits.ctypes.data)
    return hits, bad


@pytest.mark.parametrize("kind,mode", [
    ("single", "query"), ("single", "tick of many scenes"), ("instanced", "query"),
    ("instanced", "tick"), ("instanced", "tick of many scenes")])
@pytest.mark.parametrize("n,grid", [(24, 24), (40, 4), (150, 2)])
def test_helpers_have_the_state_they_use(host, kind, mode, n, grid):
    """One ray a warp, some rays a warp and more rays than lanes: the hits of the FP32 oracle and
    no read outside the scene."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    sc = _soup() if kind == "single" else _instances(_soup(), True)
    nodes, tris, _ = S.build_bvh(sc, N.BVH_MEDIUM)
    insts = None
    if kind == "instanced":
        insts = _records(sc, nodes, len(S.build_bvh(_soup(), N.BVH_MEDIUM)[0]))
    rng = np.random.default_rng(n)
    rays = np.zeros(n, N.RAY_DTYPE)
    rays["origin"] = rng.uniform(-0.5, 2.0, (n, 3))
    rays["direction"] = rng.uniform(0.2, 1.5, (n, 3)) - rays["origin"]
    rays["tmax"] = 1e7
    mixed = mode != "query"
    any_hit = (rng.uniform(size=n) < 0.4) & mixed
    if not mixed:
        rays["tmin"] = rng.uniform(0, 0.3, n)
    h, bad = _run(host, nodes, tris, insts, rays, any_hit, mixed, mode == "tick of many scenes",
                  grid)
    assert bad == 0
    o, _, _ = O.OracleScene(sc).trace_rays(rays, fp64=False, hit_dtype=N.HIT_DTYPE)
    miss = o["geometry_index"] == 0xFFFFFFFF
    assert miss.any() and not miss.all()
    assert np.array_equal(h["geometry_index"] == 0xFFFFFFFF, miss)
    c = ~miss & ~any_hit
    for f in ("t", "primitive_id", "geometry_index", "barycentrics"):
        assert np.array_equal(h[f][c].view(np.uint32), o[f][c].view(np.uint32)), f
    if kind == "instanced":
        assert np.array_equal(h["instance_id"][c], o["instance_index"][c])


def test_former_build_options(native, tmp_path):
    """A build that still sets the options of the deferred division and of the triangle records'
    axis copies, which the traversal now always has, finds the same hits."""
    fn = _build(tmp_path, ("GBPT_DEFER_UV=0", "GBPT_TRI_AXIS_COPIES=0"))
    test_helpers_have_the_state_they_use(fn, "single", "query", 40, 4)
    test_helpers_have_the_state_they_use(fn, "instanced", "tick of many scenes", 40, 4)


def _sheets():
    """Three sheets of 8 x 8 quads, one perpendicular to each axis, every triangle a two-sided
    geometry of its own in a random order: a point of a sheet lies in up to six of them."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    tris = []
    for a in range(3):
        for i in range(8):
            for j in range(8):
                q = np.zeros((4, 3))
                q[:, a] = 2.0 + 3.0 * a
                q[:, (a + 1) % 3] = np.array([i, i + 1, i + 1, i]) / 8.0
                q[:, (a + 2) % 3] = np.array([j, j, j + 1, j + 1]) / 8.0
                tris += [q[[0, 1, 2]], q[[0, 2, 3]]]
    tris = np.array(tris)[np.random.default_rng(9).permutation(len(tris))]
    n = len(tris)
    v = np.zeros(3 * n, N.VERTEX_DTYPE)
    v["position"] = tris.reshape(-1, 3)
    g = np.zeros(n, N.GEOMETRY_DTYPE)
    g["first_triangle"] = np.arange(n)
    g["triangle_count"] = 1
    g["flags"] = N.MESH_TWO_SIDED
    g["instance_mask"] = 0xFF
    m = np.zeros(1, N.MATERIAL_DTYPE)
    m["model"] = N.MATERIAL_DIFFUSE
    m["base_color_texture"] = m["alpha_texture"] = -1
    return S.SceneData(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), g, m, None), tris


def _origin_hits(two_level):
    """Rays that start on a vertex or an edge of a sheet, along either direction of its axis:
    (scene, rays, expected geometry, expected instance). The span starts at 0; of some it ends at
    +0 or -0."""
    from merian_gb300 import _native as N
    sc, tris = _sheets()
    shifts = np.zeros((1, 3))
    if two_level:
        sc = _instances(sc, False)
        shifts = np.array([np.asarray(i["object_to_world"], np.float64).reshape(3, 4)[:, 3]
                           for i in sc.instances])
    rng = np.random.default_rng(2)
    rays, geom, inst = [], [], []
    for k in range(192):
        a = k % 3
        p = np.zeros(3)
        p[a] = 2.0 + 3.0 * a
        p[(a + 1) % 3] = rng.integers(0, 9) / 8.0
        p[(a + 2) % 3] = rng.integers(0, 17) / 16.0
        s = int(rng.integers(0, len(shifts)))
        p = p + shifts[s]
        best = None
        for i, t in enumerate(shifts):
            x = p - t
            if x[a] != 2.0 + 3.0 * a:
                continue
            u, w = (a + 1) % 3, (a + 2) % 3
            c = tris[:, :, [u, w]] - x[[u, w]]
            area = [c[:, m, 0] * c[:, (m + 1) % 3, 1] - c[:, m, 1] * c[:, (m + 1) % 3, 0]
                    for m in range(3)]
            inside = (np.min(area, 0) >= 0) | (np.max(area, 0) <= 0)
            for j in np.nonzero(inside & (tris[:, 0, a] == x[a]))[0]:
                best = min(best or (int(j), i), (int(j), i))
        d = np.zeros(3)
        d[a] = 1.0 if k % 2 else -1.0
        if rng.uniform() < 0.7:
            d[(a + 1) % 3], d[(a + 2) % 3] = rng.uniform(-0.5, 0.5, 2)
        r = np.zeros(1, N.RAY_DTYPE)
        r["origin"], r["direction"] = p, d
        r["tmax"] = [1e7, 1e7, 0.0, -0.0][int(rng.integers(0, 4))]
        rays.append(r)
        geom.append(best[0])
        inst.append(best[1])
    return sc, np.concatenate(rays), np.array(geom, np.uint32), np.array(inst, np.uint32)


@pytest.mark.parametrize("kind", ["single", "instanced"])
@pytest.mark.parametrize("mode", ["query", "tick of many scenes"])
@pytest.mark.parametrize("grid", [192, 16, 1])
def test_hits_at_the_origin(host, kind, mode, grid):
    """The smallest (geometry, primitive, instance) of the triangles that hold the origin,
    whatever the sign of t = 0 and the order of the visits."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    sc, rays, geom, inst = _origin_hits(kind == "instanced")
    nodes, tris, _ = S.build_bvh(sc, N.BVH_MEDIUM)
    insts = None
    if kind == "instanced":
        insts = _records(sc, nodes, len(S.build_bvh(_sheets()[0], N.BVH_MEDIUM)[0]))
    h, bad = _run(host, nodes, tris, insts, rays, np.zeros(len(rays)), mode != "query", 1, grid)
    assert bad == 0 and (h["t"] == 0).all()
    assert np.signbit(h["t"]).any() and not np.signbit(h["t"]).all()
    assert np.array_equal(h["geometry_index"], geom)
    if kind == "instanced":
        assert np.array_equal(h["instance_id"], inst)
    else:
        w, _ = O.cwbvh_trace(nodes, tris, rays, hit_dtype=N.HIT_DTYPE)
        assert np.array_equal(w["geometry_index"], geom)
        assert np.array_equal(w["t"].view(np.uint32), h["t"].view(np.uint32))


def _special_rays(n):
    """Rays with NaN, infinite, zero and denormal components of origin and direction among
    ordinary ones, and spans with such ends."""
    from merian_gb300 import _native as N
    rng = np.random.default_rng(n)
    rays = np.zeros(n, N.RAY_DTYPE)
    rays["origin"] = rng.uniform(-0.1, 1.1, (n, 3))
    rays["direction"] = rng.normal(size=(n, 3))
    rays["tmax"] = 1e7
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-40, -1e-40, 1e-30, 3e38], np.float32)
    for f in ("origin", "direction"):
        k = rng.uniform(size=(n, 3)) < 0.12
        rays[f][k] = rng.choice(odd, k.sum())
    for f in ("tmin", "tmax"):
        k = rng.uniform(size=n) < 0.1
        rays[f][k] = rng.choice(odd, k.sum())
    return rays


def _infinite_rays(n):
    """Rays along an infinite direction: t is +0 or -0 for every triangle they meet, and the planes
    of the boxes have no slack."""
    from merian_gb300 import _native as N
    rng = np.random.default_rng(n + 1)
    rays = np.zeros(n, N.RAY_DTYPE)
    rays["origin"] = rng.uniform(0, 1, (n, 3))
    rays["direction"] = rng.normal(size=(n, 3))
    rays["direction"][np.arange(n), rng.integers(0, 3, n)] = rng.choice([-np.inf, np.inf], n)
    rays["tmin"] = rng.choice(np.array([0.0, -0.0, -1.0], np.float32), n)
    rays["tmax"] = rng.choice(np.array([1e7, 0.0, -0.0], np.float32), n)
    return rays


def _same_as_walk(h, w, any_hit):
    miss = w["geometry_index"] == 0xFFFFFFFF
    assert miss.any() and not miss.all()
    assert np.array_equal(h["geometry_index"] == 0xFFFFFFFF, miss)
    if not any_hit:
        for f in ("t", "primitive_id", "geometry_index", "barycentrics"):
            assert np.array_equal(h[f][~miss].view(np.uint32), w[f][~miss].view(np.uint32)), f


@pytest.mark.parametrize("make", [_special_rays, _infinite_rays])
@pytest.mark.parametrize("grid", [64, 3])
def test_special_values(host, make, grid):
    """The hits of the walk that visits one ray at a time, which compares the boxes' distances
    where the traversal takes signs of differences."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    nodes, tris, _ = S.build_bvh(_soup(), N.BVH_MEDIUM)
    rays = make(600)
    h, bad = _run(host, nodes, tris, None, rays, np.zeros(len(rays)), False, 0, grid)
    assert bad == 0
    w, _ = O.cwbvh_trace(nodes, tris, rays, hit_dtype=N.HIT_DTYPE)
    _same_as_walk(h, w, False)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_special_rays, _infinite_rays])
@pytest.mark.parametrize("any_hit", [False, True], ids=["closest", "any"])
def test_gpu_special_values(gpu_ctx, make, any_hit):
    import torch
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    sc = _soup()
    nodes, tris, _ = S.build_bvh(sc)
    sid = gpu_ctx.upload(sc)
    try:
        for n in (200, 20_000):
            rays = make(n)
            w, _ = O.cwbvh_trace(nodes, tris, rays, any_hit=any_hit, hit_dtype=N.HIT_DTYPE)
            r = torch.from_numpy(rays.view(np.float32).reshape(n, 8)).cuda()
            h = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            for counted in (False, True):
                gpu_ctx.trace(sid, r.data_ptr(), n, h.data_ptr(), any_hit=any_hit,
                              counted=counted)
                gpu_ctx.synchronize()
                _same_as_walk(np.frombuffer(h.cpu().numpy().tobytes(), N.HIT_DTYPE), w, any_hit)
    finally:
        gpu_ctx.destroy_scene(sid)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["single", "instanced"])
def test_gpu_hits_at_the_origin(gpu_ctx, kind):
    """The same on the GPU, counting traversal included: few rays (spread over all warps) to more
    rays than lanes."""
    import torch
    from merian_gb300 import _native as N
    sc, rays, geom, inst = _origin_hits(kind == "instanced")
    sid = gpu_ctx.upload(sc)
    try:
        for n in (1, 192, 5000, 200_000):
            k = np.arange(n) % len(rays)
            r = torch.from_numpy(rays[k].view(np.float32).reshape(n, 8)).cuda()
            h = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            for counted in (False, True):
                gpu_ctx.trace(sid, r.data_ptr(), n, h.data_ptr(), counted=counted)
                gpu_ctx.synchronize()
                g = np.frombuffer(h.cpu().numpy().tobytes(), N.HIT_DTYPE)
                assert (g["t"] == 0).all()
                assert np.array_equal(g["geometry_index"], geom[k]), (n, counted)
                if kind == "instanced":
                    assert np.array_equal(g["instance_index"], inst[k]), (n, counted)
    finally:
        gpu_ctx.destroy_scene(sid)
