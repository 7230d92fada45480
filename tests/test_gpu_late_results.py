"""Rays whose results are written with the next refill of their warp (csrc/wavefront.cu
TraceQueue): queues that mix rays without a tree, which end where they are loaded, with rays
that traverse; queues of nothing else; and queues around one and several refills."""
import numpy as np
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _without_triangles(sc):
    return sc.copy_with(indices=np.zeros((0, 3), np.int32), tri_material=np.zeros(0, np.int32),
                        tri_shading=np.zeros(0, np.uint8), lights=np.zeros(0, np.int32))


@pytest.mark.parametrize("n", [1, 20, 33, 5000, 140_000])
def test_rays_of_a_scene_without_triangles(n):
    torch = pytest.importorskip("torch")
    sc = _without_triangles(synth.spheres_grids(seed=3, tri_budget=600, env_width=16, env_height=8))
    rays = torch.randn(n, 6, device="cuda")
    tri = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    dist = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        ctx.trace_closest(ctx.upload(sc), n, rays.data_ptr(), 0.0, 3.4028235e38, tri.data_ptr(), dist.data_ptr())
        torch.cuda.synchronize()
    assert bool((tri == -1).all()) and bool((dist == -1.0).all())


@pytest.mark.parametrize("width,height,spp", [(33, 17, 3), (640, 360, 2)])
@pytest.mark.parametrize("lights", [False, True])
def test_waves_mixing_scenes_with_and_without_triangles(lights, width, height, spp):
    """The films of a batch are bit-identical to the scenes' own renders."""
    torch = pytest.importorskip("torch")
    full = synth.cornell(width=width, height=height, spp=spp, mixed=True, integrator=1, max_bounces=5,
                         env_texture=True) if lights else \
        synth.spheres_grids(seed=5, tri_budget=9000, width=width, height=height, spp=spp, max_bounces=5,
                            env_width=64, env_height=32)
    with capi.Context(0) as ctx:
        jobs = []
        for k, sc in enumerate([full, _without_triangles(full), full, _without_triangles(full)]):
            jobs.append((ctx.upload(sc), capi.camera_from_scene(sc),
                         capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=40 + k)))
        films = [torch.full((width * height * 3,), float("nan"), device="cuda") for _ in jobs]
        torch.cuda.synchronize()
        ctx.batch_render([(*j, f.data_ptr()) for j, f in zip(jobs, films)])
        torch.cuda.synchronize()
        for j, f in zip(jobs, films):
            solo = torch.full((width * height * 3,), float("nan"), device="cuda")
            torch.cuda.synchronize()
            ctx.render_device(*j, solo.data_ptr(), 0)
            torch.cuda.synchronize()
            assert bool((f.view(torch.int32) == solo.view(torch.int32)).all())
            assert float(f.mean()) > 0.0
