"""prt_build_accel while queries on a caller's stream are in flight: they read the
tree they were issued on, although the rebuild writes into the same memory."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

RAYS = 1 << 22


def _rays():
    g = torch.Generator(device="cuda").manual_seed(11)
    rays = torch.empty((RAYS, 8), device="cuda")
    rays[:, :3] = torch.rand((RAYS, 3), generator=g, device="cuda") * 24 - 12
    rays[:, 3] = 0.0
    d = torch.randn((RAYS, 3), generator=g, device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1e30
    return rays


# more streams than a context keeps track of, and queries that a graph replays
@pytest.mark.parametrize("streams,captured", [(1, False), (4, False), (33, False), (1, True)])
def test_rebuild_after_queries_on_callers_streams(small, streams, captured):
    import prt
    mesh, _ = small
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    rays = _rays()
    n = RAYS // streams
    times = 4 if streams <= 4 else 1   # a context has counters for 64 calls in flight
    ref, found = torch.empty((RAYS, 4), device="cuda"), torch.empty((RAYS, 4), device="cuda")
    # the pool hands out a stream more than once
    pool = [torch.cuda.Stream(priority=-(i & 1)) for i in range(64)]
    used = list({s.cuda_stream: s for s in pool}.values())[:streams]
    assert len(used) == streams
    for quality in (True, False, True, False):
        c.set_build_quality(quality)
        c.build()
        c.intersect(rays, ref, RAYS)
        flags = torch.empty(n, device="cuda")
        c.occluded(rays, flags, n)
        occ = torch.full((n,), 7.0, device="cuda")
        graph = torch.cuda.CUDAGraph()
        if captured:
            with torch.cuda.graph(graph, stream=used[0]):
                for _ in range(times):
                    c.intersect(rays, found, n, stream=used[0].cuda_stream)
                c.occluded(rays, occ, n, stream=used[0].cuda_stream)
        found.fill_(7.0)
        torch.cuda.synchronize()
        for k, s in enumerate(used):
            if captured:
                with torch.cuda.stream(s):
                    graph.replay()
                break
            for _ in range(times):
                c.intersect(rays[k * n:], found[k * n:], n, stream=s.cuda_stream)
            if k == 0:
                c.occluded(rays, occ, n, stream=s.cuda_stream)
        c.set_build_quality(not quality)
        c.build()
        torch.cuda.synchronize()
        assert torch.equal(found[:streams * n].view(torch.int32), ref[:streams * n].view(torch.int32))
        assert torch.equal(occ >= 0, flags >= 0)
        # and the new tree answers as the old one did
        c.intersect(rays, found, RAYS)
        assert torch.equal(found[:, 0], ref[:, 0])
    c.close()
