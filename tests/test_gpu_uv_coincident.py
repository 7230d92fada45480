"""The UV pass over coincident and degenerate triangles (the scene of test_gpu_replay_warp.py whose
oracle carries NaN weights of degenerate triangles): every value that is finite in the oracle's
pass."""
import numpy as np
import pytest

import oracle
from petrichor_gb300 import capi
from petrichor_gb300.scene_io import INTEGRATOR_PT
from test_gpu_replay_warp import ATOL, RTOL, _coincident, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textured", [False, True])
def test_finite_uvs_match(gpu_ctx, textured):
    sc = _scene(_coincident(), INTEGRATOR_PT)
    if textured:  # uvs other than zero are read at all
        rng = np.random.default_rng(2)
        sc = sc.copy_with(uvs=rng.uniform(0, 1, sc.uvs.shape).astype(np.float32))
    want = oracle.OracleScene(sc).render_aov(capi.AOV_UV, denoising_spp=2)
    sid = gpu_ctx.upload(sc)
    try:
        st = capi.settings_from_scene(sc, capi.MODE_REPLAY, denoising_spp=2)
        got = gpu_ctx.render_aov(sid, capi.camera_from_scene(sc), st, capi.AOV_UV)
    finally:
        gpu_ctx.release(sid)
    finite = np.isfinite(want)
    assert finite.mean() > 0.9
    assert np.all(np.abs(got - want)[finite] <= ATOL + RTOL * np.abs(want[finite]))
    if textured:
        assert np.abs(want[finite]).max() > 0.1
