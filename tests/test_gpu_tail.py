"""Films of waves that end in one launch (csrc/wavefront.cu TailKernel) against the staged
kernels', which profiled renders keep: the same bits, for whole waves around the path count
that picks it, and for waves whose last bounces it finishes."""
import numpy as np
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SCENES = {
    "env": lambda **k: synth.spheres_grids(seed=5, tri_budget=20_000, max_bounces=14, env_width=64, env_height=32, **k),
    "lights": lambda **k: synth.cornell(seed=5, integrator=1, max_bounces=14, mixed=True, aperture=0.05, **k),
    "simple": lambda **k: synth.cornell(seed=5, integrator=0, mixed=True, env_texture=True, **k),
}


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 7, 3), (447, 447, 1), (448, 448, 1), (640, 400, 4)])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_film_equals_the_staged_one(gpu_ctx, name, width, height, spp):
    sc = SCENES[name](width=width, height=height, spp=spp)
    sid = gpu_ctx.upload(sc)
    try:
        cam, st = capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=9)
        film = gpu_ctx.render(sid, cam, st)
        assert gpu_ctx.stats().last_device_status == 0
        staged = torch.full((height, width, 3), -1.0, device="cuda")
        torch.cuda.synchronize()
        gpu_ctx.render_profile(sid, cam, st, staged.data_ptr(), count_reference=False)
        assert np.array_equal(film.view(np.uint32), staged.cpu().numpy().view(np.uint32))
    finally:
        gpu_ctx.release(sid)
