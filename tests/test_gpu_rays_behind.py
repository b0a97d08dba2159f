"""Rays that begin behind their origin (tnear < 0): calls of few rays and single
queries find the same hits as calls of many.  Hits at negative t count in trees
with leaves of several triangles and in single queries; with one-triangle leaves
only those at t >= 0 do."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

MANY = 200000   # above 320 rays per SM


def _query(c, ray):
    import prt
    h = prt.Hit()
    r = prt.Ray.from_buffer_copy(ray.tobytes())
    assert prt.lib().prt_query_ray(c.h, C.byref(r), C.byref(h), None, None) == prt.PRT_OK
    return np.frombuffer(bytes(h), np.int32)


@pytest.mark.parametrize("tnear", [-6.0, -0.25])
def test_few_rays_equal_many_behind_the_origin(small, tnear):
    import prt
    mesh, _ = small
    g = torch.Generator(device="cuda").manual_seed(5)
    rays = torch.empty((MANY, 8), device="cuda")
    rays[:, :3] = torch.rand((MANY, 3), generator=g, device="cuda") * 24 - 12
    rays[:, 3] = tnear
    d = torch.randn((MANY, 3), generator=g, device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1e30
    host = rays[:5000].cpu().numpy()
    for leaf in (1, 2, 3):
        c = prt.Context(0)
        c.load_mesh(mesh.indices, mesh.positions)
        c.set_leaf_size(leaf)
        c.build()
        torch.cuda.synchronize()
        found = {}
        for n in (MANY, 1, 33, 5000):
            hits = torch.full((n, 4), 7.0, device="cuda")
            occ = torch.full((n,), 7.0, device="cuda")
            torch.cuda.synchronize()
            c.intersect(rays, hits, n)
            c.occluded(rays, occ, n)
            torch.cuda.synchronize()
            found[n] = hits.view(torch.int32).cpu().numpy(), occ.cpu().numpy()
        many, flags = found.pop(MANY)
        t = many[:, 0].view(np.float32)
        behind = (t < 0) & (many[:, 1] >= 0)
        assert behind[:5000].any() == (leaf > 1)
        for n, (h, o) in found.items():
            np.testing.assert_array_equal(h, many[:n])
            # which hit of an occluded ray is reported is open
            np.testing.assert_array_equal(o == -1.0, flags[:n] == -1.0)
        if leaf > 1:
            ref = many
            for i in np.flatnonzero(behind[:5000])[:20].tolist() + np.flatnonzero(~behind[:5000])[:20].tolist():
                np.testing.assert_array_equal(_query(c, host[i]), many[i])
        one = c if leaf == 1 else one
    for i in range(40):
        np.testing.assert_array_equal(_query(one, host[i]), ref[i])
