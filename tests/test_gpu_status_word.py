"""The device status of a wavefront render in a context whose first call was a ray query: the
query allocates the word that tile renders report through, which must read as clear."""
import numpy as np
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_status_is_clear_after_a_ray_query():
    sc = synth.cornell(width=8, height=8, spp=1, integrator=1)
    for _ in range(4):
        # leaves set bits in the memory the context's allocations may be given
        dirty = [torch.full((1 << k,), -1, dtype=torch.int32, device="cuda") for k in (6, 12, 18, 20, 22)]
        torch.cuda.synchronize()
        del dirty
        torch.cuda.empty_cache()
        with capi.Context(0) as ctx:
            sid = ctx.upload(sc)
            rays = torch.tensor([[0.0, -4.0, 1.0, 0.0, 1.0, 0.0]], device="cuda")
            tri = torch.zeros(1, dtype=torch.int32, device="cuda")
            dist = torch.zeros(1, device="cuda")
            torch.cuda.synchronize()
            ctx.trace_closest(sid, 1, rays.data_ptr(), 0.0, 1e30, tri.data_ptr(), dist.data_ptr())
            film = ctx.render(sid, capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT))
            assert ctx.stats().last_device_status == 0
            assert np.isfinite(film).all()
