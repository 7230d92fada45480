"""Ray queries around the sizes at which a warp's share of the rays changes and ends
(csrc/query_share.h): the hits of the same rays in another query's order, whatever the share."""
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WARPS = 28 * 152


@pytest.mark.parametrize("n", [WARPS - 1, WARPS, WARPS + 1, 2 * WARPS + 1, 17 * WARPS, 31 * WARPS, 31 * WARPS + 1])
def test_hits_do_not_depend_on_the_share(n):
    sc = synth.spheres_grids(seed=8, tri_budget=5000, env_width=16, env_height=8)
    lo, hi = torch.tensor(sc.positions.min(0), device="cuda"), torch.tensor(sc.positions.max(0), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n)
    d = torch.randn(n, 3, device="cuda", generator=g)
    rays = torch.cat([lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g), d / d.norm(dim=1, keepdim=True)], 1)
    order = torch.randperm(n, device="cuda", generator=g)
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)

        def query(r, parts):
            tri = torch.full((n,), -7, dtype=torch.int32, device="cuda")
            dist = torch.full((n,), -7.0, device="cuda")
            torch.cuda.synchronize()
            for a in range(0, n, -(-n // parts)):
                m = min(-(-n // parts), n - a)
                ctx.trace_closest(sid, m, r[a:].data_ptr(), 0.0, 3.4e38, tri[a:].data_ptr(), dist[a:].data_ptr())
            torch.cuda.synchronize()
            return tri, dist

        tri, dist = query(rays.contiguous(), 1)
        tri3, dist3 = query(rays[order].contiguous(), 3)
    assert bool((tri >= -1).all()) and 0.05 < float((tri >= 0).float().mean())
    assert bool((tri[order] == tri3).all()) and bool((dist[order] == dist3).all())
