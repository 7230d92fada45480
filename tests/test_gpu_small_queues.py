"""Closest hits of ray queues around the sizes at which the tracer spreads them over its
warps (csrc/wavefront.cu TraceQueue): one ray, part of a warp, one ray per warp of the grid
and its neighbours, a few rays per warp, full warps. Each must give the oracle's triangle
(exact) and distance (the traversal's triangle test is the reference's, bit for bit)."""
import numpy as np
import pytest

import oracle
from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 4255, 4256, 4257, 4863, 4865, 9729, 19457, 140_000])
def test_queue_sizes(n):
    torch = pytest.importorskip("torch")
    sc = synth.spheres_grids(seed=11, tri_budget=6000, n_objects=9, env_width=16, env_height=8)
    rng = np.random.default_rng(n)
    lo, hi = sc.positions.min(0), sc.positions.max(0)
    o = rng.uniform(lo, hi, (n, 3))
    d = rng.normal(size=(n, 3))
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    want_tri, want_dist = oracle.OracleScene(sc).trace(rays)
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)
        r = torch.from_numpy(rays).cuda()
        tri = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        dist = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.trace_closest(sid, n, r.data_ptr(), 0.0, 3.4028235e38, tri.data_ptr(), dist.data_ptr())
        torch.cuda.synchronize()
    tri, dist = tri.cpu().numpy(), dist.cpu().numpy()
    assert np.array_equal(tri, want_tri)
    hit = want_tri >= 0
    assert np.array_equal(dist[hit], want_dist[hit].astype(np.float32))
    assert np.all(dist[~hit] == -1.0)
