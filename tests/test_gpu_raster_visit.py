"""First hits by rasterisation against the traversal's for every form of the visit kernel
(csrc/raster_primary.cuh: groups of 8 or 32 lanes, by samples a pixel) and sample counts
around its rule, that do not divide a group, and larger than one: the same triangle and the
same distance bits for every camera ray."""
import numpy as np
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SCENES = {
    "spheres": lambda **k: synth.spheres_grids(seed=8, tri_budget=3000, n_objects=9, env_width=16, env_height=8, **k),
    "cornell": lambda **k: synth.cornell(integrator=1, **k),  # triangles wider than a segment
}


@pytest.mark.parametrize("spp", [1, 3, 7, 8, 9, 16, 17, 31, 63, 64, 65])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_rasterised_hits_equal_traced_hits(name, spp):
    w, h = 149, 67
    sc = SCENES[name](width=w, height=h, spp=spp)
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)
        cam, st = capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=3)
        out = []
        for primary in (1, 2):
            ctx.set_tuning(primary_traversal=primary)
            rays = torch.zeros(w * h * spp, 6, device="cuda")
            tri = torch.full((w * h * spp,), -7, dtype=torch.int32, device="cuda")
            dist = torch.full((w * h * spp,), -7.0, device="cuda")
            torch.cuda.synchronize()
            ctx.primary_hits(sid, cam, st, rays.data_ptr(), tri.data_ptr(), dist.data_ptr())
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in (rays, tri, dist)])
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert (out[0][1] >= 0).any()
