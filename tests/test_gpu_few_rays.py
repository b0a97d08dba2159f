"""Calls of few rays trace each with a group of lanes, calls of many with one
lane per ray: the same rays get the same hits either way, at the sizes where
warps are partly filled and where the call changes its kernel."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

MANY = 200000   # above 320 rays per SM


def _calls(c, rays, n):
    hits = torch.full((n, 4), 7.0, dtype=torch.float32, device="cuda")
    occ = torch.full((n,), 7.0, dtype=torch.float32, device="cuda")
    c.intersect(rays, hits, n)
    c.occluded(rays, occ, n)
    torch.cuda.synchronize()
    return hits.view(torch.int32).cpu().numpy(), occ.cpu().numpy()


@pytest.mark.parametrize("leaf", [1, 2, 3])
@pytest.mark.parametrize("reach", [1e30, 4.0])
def test_few_rays_equal_many(small, leaf, reach):
    import prt
    mesh, _ = small
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(leaf)
    rays = torch.empty((MANY, 8), device="cuda")
    rays[:, :3] = torch.rand((MANY, 3), generator=g, device="cuda") * 24 - 12
    rays[:, 3] = torch.rand(MANY, generator=g, device="cuda") * 0.5
    d = torch.randn((MANY, 3), generator=g, device="cuda")
    d[::7, 0] = 0.0      # rays in the planes of the axes
    d[::11, 1:] = 0.0
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True).clamp_min(1e-20)
    rays[:, 7] = reach
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.set_leaf_size(leaf)
    c.build()
    torch.cuda.synchronize()
    hits, occ = _calls(c, rays, MANY)
    assert (hits[:, 1] >= 0).any() and (hits[:, 1] < 0).any()
    for n in (1, 3, 4, 5, 31, 4 * sms, 4 * sms + 1, 16 * sms + 1, 192 * sms, 192 * sms + 1, 320 * sms, 320 * sms + 1,
              512 * sms):
        h, o = _calls(c, rays, n)
        np.testing.assert_array_equal(h, hits[:n])
        np.testing.assert_array_equal(o >= 0, occ[:n] >= 0)
        # an occluded ray's distance is some hit's, so not before the closest one
        t = h.view(np.float32)[:, 0]
        assert (o[o >= 0] >= t[o >= 0]).all()
    c.close()


def test_empty_scene_and_no_rays():
    import prt
    c = prt.Context(0)
    c.load_mesh(np.zeros((0, 3), np.int32), np.zeros((0, 3), np.float32))
    c.build()
    rays = torch.tensor([[0, 0, 0, 0, 0, 0, -1, 1e30]], dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    hits, occ = _calls(c, rays, 1)
    assert hits[0, 1] == -1 and occ[0] == -1.0
    c.intersect(rays, rays, 0)
    c.close()
