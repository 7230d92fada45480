"""Waves of interiors around the path counts up to which they run in one launch
(csrc/wavefront.cu WholeWavePaths): the films of the stages, and the launch counts that
tell which ran. The same room seen from outside keeps the larger count."""
import numpy as np
import pytest

from petrichor_gb300 import capi, synth
from petrichor_gb300.scene_io import Camera

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ONE_EACH = 152 * 4 * 128  # a path per thread of the launch


def _room(inside, **k):
    sc = synth.cornell(seed=6, spp=1, integrator=1, mixed=True, **k)
    if not inside:
        return sc
    return sc.copy_with(camera=Camera(pos=(0.05, -0.6, 1.1), view_dir=(0.2, 1.0, -0.1), fov=1.6, focus_target=None,
                                      aperture=0.0))


@pytest.mark.parametrize("inside,bounces,width,height,whole", [
    (True, 5, 304, 256, True), (True, 4, 305, 256, False), (True, 5, 500, 400, False), (True, 3, 500, 400, True),
    (False, 5, 305, 256, True), (False, 5, 500, 400, True), (False, 5, 501, 400, False)])
def test_one_launch_up_to_a_path_per_thread(gpu_ctx, inside, bounces, width, height, whole):
    assert 304 * 256 == ONE_EACH
    sc = _room(inside, max_bounces=bounces, width=width, height=height)
    sid = gpu_ctx.upload(sc)
    try:
        job = sid, capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=3)
        before = gpu_ctx.stats().kernel_launches
        film = gpu_ctx.render(*job)
        launches = gpu_ctx.stats().kernel_launches - before
        assert launches == 4 if whole else launches > 3 * (bounces + 1)
        gpu_ctx.set_tuning(tail_bounce=-1)
        staged = gpu_ctx.render(*job)
        assert np.array_equal(film.view(np.uint32), staged.view(np.uint32))
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.release(sid)
