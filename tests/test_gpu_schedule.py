"""Kernel schedules that depend on sizes: each gives the bits of the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def room(gpu_ctx):
    from merian_gb300 import scene as S
    sid = gpu_ctx.upload(S.cornell())
    yield sid, S.workload_camera("cornell-256-16spp", 64, 64)
    gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("spp", [1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 65])
@pytest.mark.parametrize("demodulate", [False, True])
def test_sample_sum_group(gpu_ctx, room, spp, demodulate):
    """The lanes that sum a pixel's samples depend on the largest sample count of the tick: alone
    (its own power of two) and beside a request of 64 samples (a whole warp), same bits."""
    from merian_gb300 import scene as S
    sid, cam = room
    p, _ = S.render_params(37, 5, spp, 4, nee=True, frame=spp, demodulate_albedo=demodulate)
    big, _ = S.render_params(9, 7, 64, 4, nee=True, frame=1)
    alone = gpu_ctx.render(sid, cam, p)
    both = gpu_ctx.render_batch([(sid, cam, p), (sid, cam, big)])
    assert np.isfinite(alone).all() and alone[:, :3].max() > 0
    assert np.array_equal(alone.view(np.uint32), both[0].view(np.uint32))


def _scenes():
    from merian_gb300 import scene as S
    from merian_gb300 import workloads as W
    import test_alpha as A
    return {"room": (S.cornell(), ((0.5, 0.5, -1.4), (0.5, 0.5, 0.0), 40.0)),
            "instanced": (W.instanced_scene(n_meshes=2, n_u=20, n_v=11, n_instances=30,
                                            n_textures=2, tex_size=16, box=10.0),
                          ((5.0, 5.0, -4.5), (5.0, 5.0, 5.0), 60.0)),
            "alpha": (A.alpha_soup(), ((0.5, 0.5, -0.6), (0.5, 0.5, 0.5), 45.0)),
            "alpha-instanced": (A.instanced(A.alpha_soup()),
                                ((2.0, 2.0, -3.0), (2.0, 2.0, 2.0), 60.0))}


@pytest.mark.parametrize("kind", ["room", "instanced", "alpha", "alpha-instanced"])
def test_primary_hits_at_ragged_sizes(gpu_ctx, kind):
    """Primary hits of images around the sizes of a warp and a block equal the FP32 oracle's bit
    for bit; the G-buffer, also at a buffer aligned to 4 bytes only, holds the same hits. A ray
    along a mesh edge (the middle row of pixels in the room) hits two triangles at one
    t: the kernels take the smaller (geometry, primitive), as the host walk of the same tree does;
    the oracle's own tree can drop one of the two, and then may only name the larger."""
    import ctypes as C
    import torch
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    from oracle import binding as O
    sc, (pos, target, fov) = _scenes()[kind]
    osc = O.OracleScene(sc)
    sid = gpu_ctx.upload(sc)
    try:
        for w, h in [(1, 1), (31, 1), (33, 1), (127, 1), (129, 1), (67, 19)]:
            cam = S.look_at(pos, target, (0.0, 1.0, 0.0), fov, 1.0)
            g = gpu_ctx.trace_primary(sid, cam, w, h)
            o, _ = osc.trace_primary(cam, w, h, fp64=False, hit_dtype=N.HIT_DTYPE)
            assert np.array_equal(g["t"].view(np.uint32), o["t"].view(np.uint32)), (w, h)
            key = [np.stack([x["instance_index"], x["geometry_index"], x["primitive_id"]], 1)
                   .astype(np.int64) for x in (g, o)]
            same = (key[0] == key[1]).all(1)
            for a, b in zip(key[0][~same], key[1][~same]):
                assert kind == "room" and tuple(a) < tuple(b)
            for f in ("instance_id", "barycentrics"):
                assert np.array_equal(g[f][same].view(np.uint32), o[f][same].view(np.uint32)), f
            buf = torch.zeros(w * h * 16 + 1, dtype=torch.int32, device="cuda")
            N.check(gpu_ctx.lib.gbpt_gbuffer(gpu_ctx.handle, sid, C.byref(cam), w, h, 0xFF,
                                             buf.data_ptr() + 4))
            gpu_ctx.synchronize()
            t = np.frombuffer(buf[1:].cpu().numpy().tobytes(), N.GBUFFER_DTYPE)
            assert np.array_equal(t["primitive_id"], g["primitive_id"])
            assert np.array_equal(t["geometry_index"],
                                  (g["geometry_index"] & 0xFFFF).astype(np.uint16))
    finally:
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("paths", [65536 - 256, 65536, 131072 - 256, 131072, 131072 + 256])
def test_sorted_vertices(gpu_ctx, paths):
    """The vertices whose shading is sorted depend on the tick's paths (a power of two and its
    neighbours): the bits of shading that is never and always sorted."""
    from merian_gb300 import scene as S
    sc = S.soup(n_triangles=20_000, n_geometries=64, env_size=(64, 32))
    sid = gpu_ctx.upload(sc)
    cam = S.look_at((0.5, 0.5, -0.6), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0), 45.0, 1.0)
    try:
        p, _ = S.render_params(256, paths // 256, 1, 6, nee=True, rr_depth=3, frame=3)
        ref = gpu_ctx.render(sid, cam, p)
        for sort in (0, 1):
            gpu_ctx.set_tuning(sort_materials=sort)
            out = gpu_ctx.render(sid, cam, p)
            assert np.array_equal(ref.view(np.uint32), out.view(np.uint32)), sort
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("kind", ["room", "instanced", "alpha", "alpha-instanced"])
def test_closest_and_shadow_rays_in_one_launch(gpu_ctx, kind):
    """A vertex's bounce rays and shadow rays share one traversal launch; profiling launches them
    apart. Same bits and ray counts, around the sizes of a warp and a block."""
    from merian_gb300 import scene as S
    sc, (pos, target, fov) = _scenes()[kind]
    if sc.env is None:
        sc.env = np.ones((8, 16, 4), np.float32)
    sid = gpu_ctx.upload(sc)
    cam = S.look_at(pos, target, (0.0, 1.0, 0.0), fov, 1.0)
    try:
        for w, h, spp in [(1, 1, 1), (31, 1, 1), (33, 1, 1), (43, 3, 1), (61, 37, 5)]:
            p, _ = S.render_params(w, h, spp, 6, nee=True, rr_depth=3, frame=w)
            a, sa = gpu_ctx.render(sid, cam, p, stats=True)
            gpu_ctx.set_profiling(1)
            b, sb = gpu_ctx.render(sid, cam, p, stats=True)
            gpu_ctx.set_profiling(0)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (w, h)
            assert (sa.rays, sa.shadow_rays, sa.trace_rays) == (sb.rays, sb.shadow_rays,
                                                                sb.trace_rays)
            assert sa.kernel_launches < sb.kernel_launches
    finally:
        gpu_ctx.set_profiling(0)
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("kind", ["room", "instanced", "alpha", "alpha-instanced"])
def test_shared_rays(gpu_ctx, kind):
    """A warp's last rays are shared out among its lanes, except in the counting traversal
    (profiling level 2): the same bits, from a single ray to more rays than lanes."""
    from merian_gb300 import scene as S
    sc, (pos, target, fov) = _scenes()[kind]
    if sc.env is None:
        sc.env = np.ones((8, 16, 4), np.float32)
    sid = gpu_ctx.upload(sc)
    cam = S.look_at(pos, target, (0.0, 1.0, 0.0), fov, 1.0)
    try:
        for w, h, spp in [(1, 1, 1), (7, 1, 1), (71, 69, 1), (97, 50, 2), (401, 397, 1)]:
            for nee in (False, True):
                p, _ = S.render_params(w, h, spp, 8, nee=nee, frame=h)
                a = gpu_ctx.render(sid, cam, p)
                gpu_ctx.set_profiling(2)
                b, _ = gpu_ctx.render(sid, cam, p, stats=True)
                gpu_ctx.set_profiling(0)
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (w, h, nee)
    finally:
        gpu_ctx.set_profiling(0)
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("kind", ["room", "instanced", "alpha", "alpha-instanced"])
@pytest.mark.parametrize("any_hit", [False, True], ids=["closest", "any"])
def test_ray_queries_equal_the_counting_traversal(gpu_ctx, kind, any_hit):
    """gbpt_trace leaves out the code a scene does not need and spreads few rays over all warps;
    gbpt_trace_counted runs the general traversal: the same hit records, first hits included."""
    import torch
    from merian_gb300 import _native as N
    sc, (pos, target, fov) = _scenes()[kind]
    side = 1.0 if sc.instances is None else (10.0 if kind == "instanced" else 4.0)
    sid = gpu_ctx.upload(sc)
    rng = np.random.default_rng(5)
    try:
        for n in (1, 31, 33, 4863, 4865, 200_001):
            rays = np.zeros(n, N.RAY_DTYPE)
            rays["origin"] = rng.uniform(0, side, (n, 3))
            rays["direction"] = rng.normal(size=(n, 3))
            rays["tmax"] = 1e7
            r = torch.from_numpy(rays.view(np.float32).reshape(n, 8)).cuda()
            h = [torch.full((n, 8), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
            torch.cuda.synchronize()
            gpu_ctx.trace(sid, r.data_ptr(), n, h[0].data_ptr(), any_hit=any_hit)
            gpu_ctx.trace(sid, r.data_ptr(), n, h[1].data_ptr(), any_hit=any_hit, counted=True)
            gpu_ctx.synchronize()
            assert torch.equal(h[0], h[1]), n
    finally:
        gpu_ctx.destroy_scene(sid)


def test_rays_with_special_values(gpu_ctx):
    """Zero directions components, infinite spans, spans with a NaN end, reversed and empty spans:
    closest and first hits as the FP32 oracle's (a NaN end: no hit)."""
    import torch
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    from oracle import binding as O
    sc = S.soup(n_triangles=5_000, n_geometries=16, env_size=None)
    osc = O.OracleScene(sc)
    sid = gpu_ctx.upload(sc)
    rng = np.random.default_rng(8)
    n = 4096
    rays = np.zeros(n, N.RAY_DTYPE)
    rays["origin"] = rng.uniform(-0.1, 1.1, (n, 3))
    rays["direction"] = rng.normal(size=(n, 3))
    rays["direction"][rng.uniform(size=(n, 3)) < 0.1] = 0.0
    rays["direction"][(rays["direction"] == 0).all(1)] = (0, 0, 1)
    kind = rng.integers(0, 5, n)
    rays["tmax"] = np.select([kind == 0, kind == 1, kind == 2], [np.inf, 0.3, -1.0], 1e7)
    rays["tmin"] = np.where(kind == 3, -0.5, 0.0)
    nan = kind == 4
    rays["tmin"][nan & (np.arange(n) % 2 == 0)] = np.nan
    rays["tmax"][nan & (np.arange(n) % 2 == 1)] = np.nan
    try:
        o, _, _ = osc.trace_rays(np.ascontiguousarray(rays[~nan]), fp64=False,
                                 hit_dtype=N.HIT_DTYPE)
        r = torch.from_numpy(rays.view(np.float32).reshape(n, 8)).cuda()
        h = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for any_hit in (False, True):
            gpu_ctx.trace(sid, r.data_ptr(), n, h.data_ptr(), any_hit=any_hit)
            gpu_ctx.synchronize()
            g = np.frombuffer(h.cpu().numpy().tobytes(), N.HIT_DTYPE)
            assert (g["geometry_index"][nan] == 0xFFFFFFFF).all()
            g = g[~nan]
            if any_hit:
                assert np.array_equal(g["geometry_index"] == 0xFFFFFFFF,
                                      o["geometry_index"] == 0xFFFFFFFF)
            else:
                for f in ("geometry_index", "primitive_id", "t"):
                    assert np.array_equal(g[f].view(np.uint32), o[f].view(np.uint32)), f
    finally:
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("kind", ["room", "instanced", "alpha", "alpha-instanced"])
@pytest.mark.parametrize("case", ["same view", "demodulated", "other mask"])
def test_primary_hits_from_a_graph_gbuffer(gpu_ctx, kind, case):
    """A renderer behind a G-buffer node of the same view takes its primary hits from the texels;
    one whose view or options differ traces them: both equal a render without a G-buffer."""
    from merian_gb300 import node
    from merian_gb300 import scene as S
    sc, (pos, target, fov) = _scenes()[kind]
    sid = gpu_ctx.upload(sc)
    try:
        for w, h, spp in [(33, 3, 1), (129, 67, 2)]:
            cam = S.look_at(pos, target, (0.0, 1.0, 0.0), fov, w / h)
            demod = case == "demodulated"
            props = {"samples per pixel": spp, "max path length": 4, "seed": 5,
                     "demodulate albedo": demod, "next event estimation": True}
            gp = {"width": w, "height": h}
            if case == "other mask":
                gp.update({str(b): False for b in range(8)})
            with node.Graph(gpu_ctx, {"nodes": {
                    "g": {"type": "GBuffer (Raytraced)", "properties": gp,
                          "outputs": ["gbuffer->r.gbuffer"]},
                    "r": {"type": "Render (Path-traced)", "properties": props}}}) as g:
                g.run(sid, cam, (w, h), 2)
                out = g.output("r.irradiance").reshape(-1, 4)
            p, _ = S.render_params(w, h, spp, 4, nee=True, frame=6, demodulate_albedo=demod)
            ref = gpu_ctx.render(sid, cam, p)
            assert np.array_equal(out.view(np.uint32), ref.view(np.uint32)), (w, h)
    finally:
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("kind", ["room", "alpha"])
@pytest.mark.parametrize("height", [1023, 1024])
def test_long_and_short_ticks(gpu_ctx, kind, height):
    """Ticks from 2^20 paths on trace with another register budget: the bits of the same frame in
    shorter ticks."""
    from merian_gb300 import scene as S
    sc, (pos, target, fov) = _scenes()[kind]
    sid = gpu_ctx.upload(sc)
    cam = S.look_at(pos, target, (0.0, 1.0, 0.0), fov, 1.0)
    try:
        p, _ = S.render_params(1024, height, 1, 4, nee=True, frame=2)
        a = gpu_ctx.render(sid, cam, p)
        gpu_ctx.set_tuning(wave_paths=1 << 19)
        b = gpu_ctx.render(sid, cam, p)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.destroy_scene(sid)


def test_sorted_few_pixels_of_many_samples(gpu_ctx):
    """A pixel's sort key serves all its samples: requests of few pixels and many samples, around
    the sizes of the sort's tiles and several to a tick, give the bits of unsorted shading, and
    the primary pass does not grow with the samples of a pixel (its time with the sample sums is
    that of unsorted shading; a factor of 2 covers the timer)."""
    from merian_gb300 import scene as S
    sid = gpu_ctx.upload(S.soup(n_triangles=20_000, n_geometries=64, env_size=(64, 32)))
    cam = S.look_at((0.5, 0.5, -0.6), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0), 45.0, 1.0)
    jobs, keep = [], []
    for px, spp in [(1, 1), (1, 2047), (3, 2049), (5, 4096), (37, 33), (2, 70_001)]:
        pix = np.random.default_rng(px).choice(64 * 64, px, replace=False).astype(np.uint32)
        p, k = S.render_params(64, 64, spp, 4, nee=True, rr_depth=3, frame=spp, pixels=pix)
        jobs.append((sid, cam, p))
        keep.append((pix, k))
    pix = np.arange(64, dtype=np.uint32) * 61
    many, k = S.render_params(64, 64, 1 << 16, 2, nee=False, frame=1, pixels=pix)
    try:
        outs, other = [], []
        for sort in (0, 1, -1):
            gpu_ctx.set_tuning(sort_materials=sort)
            outs.append([gpu_ctx.render(*j) for j in jobs] + gpu_ctx.render_batch(jobs))
            gpu_ctx.set_profiling(1)
            other.append(min(gpu_ctx.render(sid, cam, many, stats=True)[1].other_ms
                             for _ in range(3)))
            gpu_ctx.set_profiling(0)
        for o in outs[1:]:
            assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32))
                       for a, b in zip(outs[0], o))
        assert max(other[1:]) < 2 * other[0], other
    finally:
        gpu_ctx.set_profiling(0)
        gpu_ctx.set_tuning()
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("spp", [1, 8, 33, 7 * 32, 8 * 32 - 1, 8 * 32, 8 * 32 + 1, 9 * 32 - 1,
                                 16 * 32 + 5])
def test_sample_sum_of_equal_samples(gpu_ctx, spp):
    """The samples of a pixel that sees the environment are equal: their sum is NumPy's in the
    kernel's order (each lane its samples one after the other, several loads in flight or not,
    then the tree), to the last bit."""
    import test_gpu_errors as E
    from merian_gb300 import scene as S
    sc = E.quad()
    sc.env = np.tile(np.array([0.1, 0.7, 0.3, 1.0], np.float32), (8, 16, 1))
    sid = gpu_ctx.upload(sc)
    cam = S.look_at((0, 0, 0), (0, 0, -1), (0, 1, 0), 60.0, 1.0)
    try:
        p, _ = S.render_params(3, 3, 1, 1, frame=2)
        v = gpu_ctx.render(sid, cam, p)[:, :3]
        p, _ = S.render_params(3, 3, spp, 1, frame=2)
        out = gpu_ctx.render(sid, cam, p)
    finally:
        gpu_ctx.destroy_scene(sid)
    fma = lambda a, b, c: np.float32(np.longdouble(a) * np.longdouble(b) + np.longdouble(c))
    group = 1
    while group < min(spp, 32):
        group *= 2
    for px in range(9):
        r, g, b = v[px]
        lum = fma(b, np.float32(0.114), fma(g, np.float32(0.587), np.float32(0.299) * r))
        lanes = np.zeros((group, 4), np.float32)
        for lane in range(group):
            for _ in range(lane, spp, group):
                lanes[lane, :3] += v[px]
                lanes[lane, 3] = fma(lum, lum, lanes[lane, 3])
        off = group // 2
        while off:
            lanes = lanes + lanes[np.arange(group) ^ off]
            off //= 2
        want = lanes[0] * (np.float32(1.0) / np.float32(spp))
        assert np.array_equal(out[px].view(np.uint32), want.view(np.uint32)), px


def test_sample_sum_of_one_pixel(gpu_ctx, room):
    """2^20 samples of a pixel with the primary pass in 5 ms: with one load after the other in
    flight their sum takes more than twice that, with eight 2.7 ms."""
    from merian_gb300 import scene as S
    sid, cam = room
    pix = np.array([64 * 30 + 31], np.uint32)
    p, k = S.render_params(64, 64, 1 << 20, 2, frame=4, pixels=pix)
    try:
        gpu_ctx.set_profiling(1)
        ms = min(gpu_ctx.render(sid, cam, p, stats=True)[1].other_ms for _ in range(3))
    finally:
        gpu_ctx.set_profiling(0)
    assert ms < 5


@pytest.mark.parametrize("touched", ["none", "first half", "every other page", "all"])
def test_host_outputs_in_any_pages(gpu_ctx, room, touched):
    """Host outputs whose pages are absent, partly or wholly present, at the end of a mapping and
    not at a page's start: the image, and nothing beside it."""
    import ctypes as C
    import mmap
    from merian_gb300 import _native as N
    from merian_gb300 import scene as S
    sid, cam = room
    w = h = 160  # 400 KB
    p, _ = S.render_params(w, h, 1, 2, frame=9)
    ref = gpu_ctx.render(sid, cam, p)
    size = -(-(ref.nbytes + 4096) // mmap.PAGESIZE) * mmap.PAGESIZE
    with mmap.mmap(-1, size) as m:
        buf = np.frombuffer(m, np.uint8)
        at = size - ref.nbytes
        if touched != "none":
            step = mmap.PAGESIZE * (2 if touched == "every other page" else 1)
            buf[:size // 2 if touched == "first half" else size:step] = 7
        before = buf[:at].copy() if touched != "none" else np.zeros(at, np.uint8)
        out = C.c_void_p(buf.ctypes.data + at)
        N.check(gpu_ctx.lib.gbpt_render(gpu_ctx.handle, sid, C.byref(cam), C.byref(p), out, None))
        assert np.array_equal(buf[at:], ref.view(np.uint8).reshape(-1))
        assert np.array_equal(buf[:at], before)
        del buf


def test_autotuner_leaves_out_the_postponement(gpu_ctx):
    """trace_postpone_lanes has no effect: the autotuner renders none of its five values, answers
    the default and gives the best time so far for them."""
    from merian_gb300 import scene as S
    sid = gpu_ctx.upload(S.soup(n_triangles=3_000, n_geometries=8, env_size=(32, 16)))
    cam = S.look_at((0.5, 0.5, -0.6), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0), 45.0, 1.0)
    p, _ = S.render_params(96, 96, 3, 7, nee=True, rr_depth=2, frame=1)
    try:
        t, ms = gpu_ctx.autotune(sid, cam, p)
        assert len(ms) == 21 and t.trace_postpone_lanes == 6
        assert ms[13:18] == [ms[13]] * 5 and ms[13] in ms[:13]
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.destroy_scene(sid)


@pytest.mark.parametrize("differs", ["nothing", "position", "jitter", "far plane", "scene"])
def test_graph_gbuffer_of_another_view(gpu_ctx, tmp_path, differs):
    """A renderer takes primary hits from its G-buffer only when that was traced for the same
    scene and camera: here the G-buffer's come from a scene file, the renderer's from the graph's
    call. Always the frame of the renderer's own view."""
    from test_gltf import build_scene
    from merian_gb300 import node
    from merian_gb300 import scene as S
    path, _ = build_scene(tmp_path, "glb")
    sc, cam, _, _ = S.load_gltf(path)
    w, h = 72, 48
    other = gpu_ctx.upload(sc)  # the file's scene gets the next id
    if differs == "position":
        cam.position[0] += 0.125
    elif differs == "jitter":
        cam.jitter[0] = 0.375
    elif differs == "far plane":
        cam.far_plane = 2.0
    try:
        with node.Graph(gpu_ctx, {"nodes": {
                "s": {"type": "GLTF Scene", "properties": {"file": str(path)},
                      "outputs": ["scene->g.scene"]},
                "g": {"type": "GBuffer (Raytraced)", "properties": {"width": w, "height": h},
                      "outputs": ["gbuffer->r.gbuffer"]},
                "r": {"type": "Render (Path-traced)", "properties": {"samples per pixel": 2}}}}) as g:
            g.run(other if differs == "scene" else other + 1, cam, (w, h), 2)
            out = g.output("r.irradiance").reshape(-1, 4)
        p, _ = S.render_params(w, h, 2, 5, frame=1)
        ref = gpu_ctx.render(other, cam, p)
        assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))
    finally:
        gpu_ctx.destroy_scene(other)
