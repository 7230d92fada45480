"""Ray queries on several streams at once: each gives the hits that it gives alone. Sizes on
both sides of the one from which the warps fetch from a counter (csrc/query_share.h)."""
import pytest

from petrichor_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [700, 31 * 28 * 152, 31 * 28 * 152 + 1, 200_000])
def test_concurrent_queries(n):
    sc = synth.spheres_grids(seed=4, tri_budget=20_000, env_width=16, env_height=8)
    lo, hi = torch.tensor(sc.positions.min(0), device="cuda"), torch.tensor(sc.positions.max(0), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n)
    queries = 40  # more than a context has counters
    org = lo + (hi - lo) * torch.rand(queries, n, 3, device="cuda", generator=g)
    d = torch.randn(queries, n, 3, device="cuda", generator=g)
    rays = torch.cat([org, d / d.norm(dim=-1, keepdim=True)], -1).contiguous()
    tri = torch.full((2, queries, n), -7, dtype=torch.int32, device="cuda")
    dist = torch.full((2, queries, n), -7.0, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)
        for alone in (1, 0):
            for q in range(queries):
                ctx.trace_closest(sid, n, rays[q].data_ptr(), 0.0, 3.4e38, tri[alone, q].data_ptr(),
                                  dist[alone, q].data_ptr(), streams[q % 4].cuda_stream)
                if alone:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
    assert bool((tri[0] == tri[1]).all()) and bool((dist[0] == dist[1]).all())
    assert bool((tri[1] >= -1).all()) and 0.05 < float((tri[1] >= 0).float().mean())


def test_captured_query_replays():
    """A captured query, replayed beside direct ones on another stream."""
    n = 150_000
    sc = synth.spheres_grids(seed=4, tri_budget=20_000, env_width=16, env_height=8)
    rays = torch.randn(n, 6, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    tri = torch.full((3, n), -7, dtype=torch.int32, device="cuda")
    dist = torch.full((3, n), -7.0, device="cuda")
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        sid = ctx.upload(sc)

        def query(k, s):
            ctx.trace_closest(sid, n, rays.data_ptr(), 0.0, 3.4e38, tri[k].data_ptr(), dist[k].data_ptr(), s.cuda_stream)

        query(0, other)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            query(1, side)
        for _ in range(20):
            tri[1:].fill_(-7)
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                graph.replay()
            query(2, other)
            torch.cuda.synchronize()
            assert bool((tri[1] == tri[0]).all()) and bool((tri[2] == tri[0]).all())
            assert bool((dist[1] == dist[0]).all()) and bool((dist[2] == dist[0]).all())
