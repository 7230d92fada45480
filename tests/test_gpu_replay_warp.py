"""Replay and AOV passes (one warp per tile, csrc/replay.cu TraverseWarp) on trees at the
edges of the warp's traversal: a chain deeper than its shared-memory stack, leaves of more
triangles than a warp has lanes (coincident triangles, whose ties the first one wins),
degenerate triangles, a single triangle; against the oracle."""
import math

import numpy as np
import pytest

import oracle
from petrichor_gb300 import capi, scene_io, synth
from petrichor_gb300.scene_io import (Camera, Environment, Material, Scene, Settings, MAT_GLASS, MAT_LAMBERT,
                                      INTEGRATOR_PT, INTEGRATOR_SIMPLE)

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-4, 1e-6  # the replay films' tolerance (FP32 radiance)


def _scene(tris, integrator, width=21, height=18, spp=2, tile=8):
    P = np.asarray(tris, np.float64).reshape(-1, 3)
    b = synth._Builder()
    b.add(P, np.arange(P.shape[0]).reshape(-1, 3), 0, scene_io.SHADING_FLAT)
    pos, nrm, uv, idx, tm, sh = b.arrays()
    tm = (np.arange(len(idx)) % 2).astype(np.int32)
    mats = [Material(MAT_LAMBERT, color=(0.6, 0.5, 0.4)), Material(MAT_GLASS, ior=1.5)]
    cam = Camera(pos=(0.0, 0.0, 0.0), view_dir=(1.0, 0.0, 0.0), fov=math.radians(50.0), aperture=0.0)
    st = Settings(width=width, height=height, spp=spp, max_bounces=4, integrator=integrator, tile_width=tile,
                  tile_height=tile)
    return Scene(pos, nrm, uv, idx, tm, sh, np.zeros(0, np.int32), mats, cam,
                 Environment(base_color=(1.0, 0.9, 0.8), texture=None), st)


def _facing(x, s):
    return [[x, -s, -s], [x, s, -0.2 * s], [x, -0.1 * s, s]]


def _chain():  # distances growing 13-fold: each split takes one triangle off, 30 levels
    return [_facing(float(np.float32(2.0 ** -62 * 13.0 ** i)), 0.35 * float(2.0 ** -62 * 13.0 ** i)) for i in range(34)]


def _coincident():
    flat = [[[2.0, 0.1, 0.1]] * 3, [[2.5, -0.3, 0.0], [2.5, 0.0, 0.0], [2.5, 0.3, 0.0]]]
    return [_facing(4.0, 1.5)] * 70 + flat + [_facing(5.0, 3.0)] * 3


SCENES = {"chain": _chain, "coincident": _coincident, "single": lambda: [_facing(3.0, 1.0)]}


@pytest.mark.parametrize("integrator", [INTEGRATOR_SIMPLE, INTEGRATOR_PT])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_replay_and_aov_match_oracle(gpu_ctx, name, integrator):
    sc = _scene(SCENES[name](), integrator)
    bounds, ints, _, height = capi.bvh_build(sc.positions, sc.indices)
    if name == "chain":
        assert height > 24  # more pending entries than the shared-memory stack holds
    if name == "coincident":
        assert (ints[:, 3] - ints[:, 2])[ints[:, 4] == 1].max() > 64
    o = oracle.OracleScene(sc)
    ref, _ = o.render()
    sid = gpu_ctx.upload(sc)
    try:
        cam, st = capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_REPLAY, denoising_spp=2)
        film = gpu_ctx.render(sid, cam, st)
        assert gpu_ctx.stats().last_device_status == 0
        assert np.all(np.abs(film - ref) <= ATOL + RTOL * np.abs(ref))
        for aov in (capi.AOV_UV, capi.AOV_DENOISING_ALBEDO, capi.AOV_DENOISING_NORMAL):
            got = gpu_ctx.render_aov(sid, cam, st, aov)
            want = o.render_aov(aov, denoising_spp=2)
            if name == "coincident" and aov == capi.AOV_UV:
                continue  # a degenerate triangle's uv weights are NaN; a scene without uvs reads as 0 here
            assert np.array_equal(np.isnan(got), np.isnan(want))
            ok = np.isnan(want) | (np.abs(got - want) <= ATOL + RTOL * np.abs(want))
            assert np.all(ok)
    finally:
        gpu_ctx.release(sid)
