"""The device traversal run on the host (traversal_host.cpp): rays shared among a warp's lanes.

Unset lane state holds a pattern and reads outside the scene's arrays are counted, so these tests
see on the CPU what a helper lane that never loaded a ray of its own works with.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import binding as O


@pytest.fixture(scope="module")
def host(native, tmp_path_factory):
    from merian_gb300 import build as B
    lib = tmp_path_factory.mktemp("traversal") / "libtraversal.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ftrivial-auto-var-init=pattern",
                    "-ffp-contract=off", "-fPIC", "-shared", "-I", str(B.INCLUDE), "-I",
                    str(B.CSRC), "-I", str(B._cuda_home() / "include"),
                    str(ROOT / "tests" / "traversal_host.cpp"), "-o", str(lib)], check=True)
    fn = C.CDLL(str(lib)).traversal_host
    fn.restype = C.c_int64
    vp, u32, u64, i32 = C.c_void_p, C.c_uint32, C.c_uint64, C.c_int
    fn.argtypes = [vp, u64, vp, u64, vp, u64, i32, i32, vp, vp, u32, u32, u32, vp]
    return fn


def _soup():
    from merian_gb300 import scene as S
    return S.soup(n_triangles=4000, n_geometries=8, env_size=None)


def _instances():
    """Eight overlapping instances of one BLAS: translations and a permutation of the axes, whose
    inverses are exact."""
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    sc = _soup()
    rng = np.random.default_rng(4)
    inst = np.zeros(8, N.INSTANCE_DTYPE)
    for k in range(8):
        m = np.zeros((3, 4), np.float32)
        m[:, :3] = np.roll(np.eye(3), k, axis=0)
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
    sc = _soup() if kind == "single" else _instances()
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
