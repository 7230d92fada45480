"""Scene records formed on the device (csrc/scene_records.cu): optional arrays left out equal
their defaults spelled out, a leaf longer than a thread marks by itself, a scene without
triangles, and both BVH builders (whose arrays reach the kernels by different routes)."""
import ctypes

import numpy as np
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu


class _Without:
    """A library handle whose pt_scene_upload drops the optional arrays."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        if name != "pt_scene_upload":
            return getattr(self._lib, name)

        def upload(h, desc, sid):
            d = desc._obj
            d.normals = d.uvs = d.tri_shading = None
            return self._lib.pt_scene_upload(h, ctypes.byref(d), sid)
        return upload


def _film(ctx, sc, mode=capi.MODE_REPLAY):
    sid = ctx.upload(sc)
    try:
        return ctx.render(sid, capi.camera_from_scene(sc), capi.settings_from_scene(sc, mode))
    finally:
        ctx.release(sid)


@pytest.mark.parametrize("builder", [capi.BVH_BUILDER_HOST, capi.BVH_BUILDER_DEVICE])
@pytest.mark.parametrize("textured", [False, True])
def test_left_out_arrays_are_their_defaults(builder, textured):
    make = synth.textured_spheres if textured else synth.spheres_grids
    sc = make(tri_budget=1500, width=40, height=23, spp=2, env_width=33, env_height=17)
    n, t = sc.positions.shape[0], sc.indices.shape[0]
    plain = sc.copy_with(normals=np.tile(np.float32([0, 0, 1]), (n, 1)), uvs=np.zeros((n, 3), np.float32),
                         tri_shading=np.zeros(t, np.uint8))
    with capi.Context(0) as ctx:
        ctx.set_bvh_builder(builder)
        for mode in (capi.MODE_REPLAY, capi.MODE_WAVEFRONT):
            want = _film(ctx, plain, mode)
            lib, ctx.L = ctx.L, _Without(ctx.L)
            got = _film(ctx, sc, mode)
            ctx.L = lib
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
            assert got.mean() > 0


def test_builders_agree_on_long_leaves_and_empty_scenes():
    sc = synth.cornell(width=24, height=24, spp=2, integrator=1, env_texture=True)
    idx = np.concatenate([sc.indices[:10]] + [sc.indices[10:11]] * 300 + [sc.indices[11:]])
    mat = np.concatenate([sc.tri_material[:10]] + [sc.tri_material[10:11]] * 300 + [sc.tri_material[11:]])
    sh = np.concatenate([sc.tri_shading[:10]] + [sc.tri_shading[10:11]] * 300 + [sc.tri_shading[11:]])
    long = sc.copy_with(indices=idx, tri_material=mat, tri_shading=sh, lights=np.zeros(0, np.int32))
    empty = sc.copy_with(indices=sc.indices[:0], tri_material=sc.tri_material[:0], tri_shading=sc.tri_shading[:0],
                         lights=np.zeros(0, np.int32))
    with capi.Context(0) as ctx:
        for scene in (long, empty):
            films = []
            for builder in (capi.BVH_BUILDER_HOST, capi.BVH_BUILDER_DEVICE):
                ctx.set_bvh_builder(builder)
                films += [_film(ctx, scene, m) for m in (capi.MODE_REPLAY, capi.MODE_WAVEFRONT)]
            assert np.array_equal(films[0].view(np.uint32), films[2].view(np.uint32))
            assert np.array_equal(films[1].view(np.uint32), films[3].view(np.uint32))
