"""The environment sampler's outcome table (csrc/env_row.h, pt_device.cuh EnvSampleLit) at the
edges of its rule: one-row and one-column maps, the largest tabled height, the next one (formed
per sample) and sizes that are not powers of two; replay films against the oracle, and the
throughput path's mean against the replay's."""

import numpy as np
import pytest

import oracle
from petrichor_gb300 import capi, synth
from petrichor_gb300.scene_io import Environment

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-4, 1e-6  # the replay films' tolerance


@pytest.mark.parametrize("height,width", [(1, 1), (1, 4), (2, 1), (32, 64), (30, 64), (8192, 2), (16384, 2)])
def test_replay_matches_oracle(gpu_ctx, height, width):
    rng = np.random.default_rng(height)
    sc = synth.cornell(width=32, height=24, spp=2, mixed=True, integrator=1, max_bounces=4)
    env = Environment(base_color=(0.9, 1.0, 0.8), z_rotation=0.7,
                      texture=rng.uniform(0.2, 2.0, (height, width, 3)).astype(np.float32))
    sc = sc.copy_with(env=env, lights=np.zeros(0, np.int32))
    ref, _ = oracle.OracleScene(sc).render()
    sid = gpu_ctx.upload(sc)
    try:
        cam = capi.camera_from_scene(sc)
        film = gpu_ctx.render(sid, cam, capi.settings_from_scene(sc, capi.MODE_REPLAY))
        assert gpu_ctx.stats().last_device_status == 0
        assert np.all(np.abs(film - ref) <= ATOL + RTOL * np.abs(ref))
        a, b = (gpu_ctx.render(sid, cam, capi.settings_from_scene(sc, m, seed=4, spp=256))
                for m in (capi.MODE_WAVEFRONT, capi.MODE_REPLAY))
        # two estimates of one image mean from 196,608 samples each; sigma of a sample's mean
        # from the pixels' spread
        sigma = np.sqrt((a.reshape(-1, 3).var(0) + b.reshape(-1, 3).var(0)) / (32 * 24)).max()
        assert np.all(np.abs(a.mean((0, 1)) - b.mean((0, 1))) <= 5 * sigma)
    finally:
        gpu_ctx.release(sid)
