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
