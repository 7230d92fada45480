"""Ray queries with axis-parallel directions (two components exactly zero, of either sign, or too
small for their reciprocal): the oracle's triangle (exact) and distance (bit for bit), in
a box of axis-parallel walls around zero, over spheres and over terrain."""
import numpy as np
import pytest

import oracle
from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SCENES = {
    "box": lambda: synth.cornell(mixed=True, integrator=1),
    "spheres": lambda: synth.spheres_grids(seed=11, tri_budget=6000, n_objects=9, env_width=16, env_height=8),
    "terrain": lambda: synth.terrain_rocks(seed=4, terrain_n=40, n_rocks=20, rock_tris=60, env_width=16, env_height=8),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_hits_equal_the_oracles(name):
    sc = SCENES[name]()
    rng = np.random.default_rng(5)
    n = 12_000
    lo, hi = sc.positions.min(0), sc.positions.max(0)
    span = hi - lo
    o = rng.uniform(lo - 0.1 * span, hi + 0.1 * span, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    small = np.array([0.0, -0.0, 1e-45, -1e-40], np.float32)
    axis = rng.integers(0, 3, n)
    for k in (1, 2):
        d[np.arange(n), (axis + k) % 3] = small[rng.integers(0, 4, n)]
    d /= np.linalg.norm(d.astype(np.float64), axis=1, keepdims=True).astype(np.float32)
    rays = np.concatenate([o, d], 1).astype(np.float32)
    want_tri, want_dist = oracle.OracleScene(sc).trace(rays)
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)
        r = torch.from_numpy(rays).cuda()
        tri = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        dist = torch.full((n,), -7.0, device="cuda")
        torch.cuda.synchronize()
        ctx.trace_closest(sid, n, r.data_ptr(), 0.0, 3.4028235e38, tri.data_ptr(), dist.data_ptr())
        torch.cuda.synchronize()
    tri, dist = tri.cpu().numpy(), dist.cpu().numpy()
    hit = want_tri >= 0
    assert hit.mean() > 0.1
    assert np.array_equal(tri, want_tri)
    assert np.array_equal(dist[hit], want_dist[hit].astype(np.float32)) and np.all(dist[~hit] == -1.0)
