"""Waves that keep all their stages (pt_tuning.tail_bounce = -1). By default a small wave runs in
one launch (csrc/wavefront.cu TailKernel), and so would the launch configurations of
test_gpu_tuning.py, whose images are small: here they run the stage kernels, which the counts of
launches show, with the films of the default. The checked build runs them too."""
import os
import subprocess
import sys

import numpy as np
import pytest

from petrichor_gb300 import capi, synth
from test_gpu_tuning import _render, _scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CONFIGS = [dict(), dict(use_graphs=0), dict(blocks_per_sm=4, band_rows=16), dict(blocks_per_sm=1, use_graphs=0),
           dict(blocks_per_sm=8), dict(band_rows=1, wave_paths=3000), dict(sort_rays=1),
           dict(primary_traversal=1), dict(primary_traversal=1, use_graphs=0, wave_paths=3000),
           dict(primary_traversal=2), dict(primary_traversal=2, use_graphs=0, wave_paths=3000)]


@pytest.fixture(scope="module")
def staged():
    with capi.Context() as ctx:
        jobs = {}
        for name, sc in _scenes().items():
            jobs[name] = (ctx.upload(sc), capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=7))
        yield ctx, jobs


def _counted(ctx, job):
    before = ctx.stats().kernel_launches
    film = _render(ctx, *job)
    return film, ctx.stats().kernel_launches - before


@pytest.mark.parametrize("name", ["pt", "simple", "tris", "raster", "inside", "overflow"])
def test_staged_films_equal_the_default(staged, name):
    ctx, jobs = staged
    job = jobs[name]
    ctx.set_tuning()
    ref, _ = _counted(ctx, job)
    assert np.isfinite(ref).all()
    for cfg in CONFIGS:
        ctx.set_tuning(tail_bounce=-1, **cfg)
        for _ in range(2):  # the second render replays the captured graph
            film, launches = _counted(ctx, job)
            assert np.array_equal(film.view(np.uint32), ref.view(np.uint32)), cfg
        # raygen, at least extend and shade per bounce (four bounces at a time where polled), sums, film
        bounces = 4 if name == "simple" else job[2].max_bounces + 1
        per = 2 if name == "simple" else 6 if cfg.get("sort_rays") else 3
        raster = 4 if cfg.get("primary_traversal") == 2 and name == "overflow" else 0
        assert launches >= 3 + per * bounces + raster, (cfg, launches)
    ctx.set_tuning()


def test_small_waves_run_in_one_launch_by_default(staged):
    ctx, jobs = staged
    for name in ("pt", "simple", "tris", "inside", "overflow"):
        ctx.set_tuning()
        assert _counted(ctx, jobs[name])[1] == 4  # raygen, paths, sums, film
        ctx.set_tuning(tail_bounce=2)  # an explicit bounce keeps the ones before it staged
        assert _counted(ctx, jobs[name])[1] >= 3 + 2 * 2 + (name != "simple")
    ctx.set_tuning()


def test_a_grid_takes_effect_after_the_default_was_captured(staged):
    """A captured sequence is used again only for the same grids of all stages."""
    ctx, jobs = staged
    films = []
    for cfg in (dict(), dict(blocks_per_sm=8), dict(blocks_per_sm=7), dict()):
        ctx.set_tuning(tail_bounce=-1, **cfg)
        films.append(_render(ctx, *jobs["pt"]))
    ctx.set_tuning()
    assert all(np.array_equal(f.view(np.uint32), films[0].view(np.uint32)) for f in films)


def test_batches_raster_and_trace_alike_in_stages(staged):
    ctx, jobs = staged
    names = ["pt", "raster", "tris", "overflow", "simple"]
    films = {}
    for traversal in (0, 1, 2):
        ctx.set_tuning(tail_bounce=-1, primary_traversal=traversal)
        out = [torch.full((jobs[n][2].width * jobs[n][2].height * 3,), float("nan"), device="cuda") for n in names]
        torch.cuda.synchronize()
        before = ctx.stats().kernel_launches
        ctx.batch_render([(*jobs[n], f.data_ptr()) for n, f in zip(names[:4], out)])
        torch.cuda.synchronize()
        # raygen, eight bounces of three, sums and film; four more where units are rasterised
        assert ctx.stats().kernel_launches - before >= 3 + 3 * 8 + (0 if traversal == 1 else 4)
        ctx.batch_render([(*jobs[n], f.data_ptr()) for n, f in zip(names, out)])  # polled: a job without a limit
        torch.cuda.synchronize()
        films[traversal] = [f.cpu().numpy() for f in out]
    ctx.set_tuning()
    for n, a, b, c in zip(names, *films.values()):
        solo = _render(ctx, *jobs[n])
        for f in (a, b, c):
            assert np.array_equal(f.view(np.uint32), solo.view(np.uint32)), n


def test_tail_bounce_takes_minus_one(staged):
    ctx, _ = staged
    ctx.set_tuning(tail_bounce=-1)
    assert ctx.get_tuning().tail_bounce == -1
    ctx.set_tuning()


SCRIPT = r"""
import sys
import numpy as np
import torch
sys.path.insert(0, ROOT)
sys.path.insert(0, ROOT + "/tests")
from petrichor_gb300 import capi, _build
from test_gpu_tuning import _render, _scenes
L = capi.load()
assert L._name.startswith(_build.CHECK_DIR), L._name
with capi.Context() as ctx:
    jobs = []
    for name, sc in _scenes().items():
        job = (ctx.upload(sc), capi.camera_from_scene(sc), capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed=7))
        films = []
        for cfg in (dict(), dict(primary_traversal=1), dict(primary_traversal=2), dict(sort_rays=1), dict(wave_paths=3000)):
            for tail in (0, -1):
                ctx.set_tuning(tail_bounce=tail, **cfg)
                film = np.full((job[2].height, job[2].width, 3), np.nan, np.float32)
                films.append(ctx.render(*job, film).copy())
                assert ctx.stats().last_device_status == 0, (name, cfg, tail, ctx.stats().last_device_status)
        assert all(np.array_equal(f.view(np.uint32), films[0].view(np.uint32)) for f in films), name
        jobs.append((*job, torch.empty(job[2].width * job[2].height * 3, device="cuda")))
    for traversal in (0, 2):
        ctx.set_tuning(tail_bounce=-1, primary_traversal=traversal)
        ctx.batch_render([(*j[:3], j[3].data_ptr()) for j in jobs])
        torch.cuda.synchronize()
        ctx.render(*jobs[0][:3])
        assert ctx.stats().last_device_status == 0
print("checked stages clean")
"""


def test_checked_build_runs_the_stages_without_bounds_errors():
    env = dict(os.environ, PT_GB300_CHECKED="1")
    r = subprocess.run([sys.executable, "-c", SCRIPT.replace("ROOT", repr(ROOT))], env=env, capture_output=True, text=True,
                       timeout=1500, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "checked stages clean" in r.stdout
