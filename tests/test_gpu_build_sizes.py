"""The SAH build at the sizes where its phases meet: one warp window (32
triangles), one subtree (256), one chunk (2048) and tasks of several chunks,
and rebuilds into the block of an earlier build.  Every triangle is in one leaf,
and closest hits equal those of the low-quality (Morton) tree."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _soup(n, kind, seed=11):
    rng = np.random.default_rng(seed + n)
    c = rng.uniform(-1, 1, (n, 1, 3))
    if kind == "clustered":
        # most centroids in few places: bins that separate nothing, uneven splits
        c = c * np.where(rng.random((n, 1, 1)) < 0.8, 1e-3, 1.0) + rng.integers(0, 2, (n, 1, 1))
    if kind == "flat":
        c[..., 1] = 0.0
    pos = (c + rng.uniform(-1, 1, (n, 3, 3)) * 0.5 * n ** -0.4).astype(np.float32)
    if kind == "flat":
        pos[..., 1] = 0.25
    return pos.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(n, 3)


def _hits(c, rays):
    hits = torch.empty((len(rays), 4), dtype=torch.float32, device="cuda")
    c.intersect(rays, hits, len(rays))
    torch.cuda.synchronize()
    return hits[:, 0].cpu().numpy(), hits.view(torch.int32)[:, 1].cpu().numpy()


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 255, 256, 257, 513, 2047, 2048, 2049, 4097, 9001, 70001])
@pytest.mark.parametrize("kind", ["uniform", "clustered", "flat"])
def test_build_sizes(n, kind):
    import prt
    pos, idx = _soup(n, kind)
    g = torch.Generator(device="cuda").manual_seed(n)
    m = 4096
    rays = torch.empty((m, 8), device="cuda")
    rays[:, :3] = torch.rand((m, 3), generator=g, device="cuda") * 3 - 1
    rays[:, 3] = 0
    d = torch.randn((m, 3), generator=g, device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1e30
    torch.cuda.synchronize()
    c = prt.Context(0)
    c.load_mesh(idx, pos)
    found = []
    for high in (True, False, True):   # the third build reuses the block of the second
        c.set_build_quality(high)
        c.build()
        _, tris = c.read_accel()
        prims = tris[:, 3].view(np.int32)
        np.testing.assert_array_equal(np.sort(prims), np.arange(n))
        np.testing.assert_array_equal(tris[:, 4:7], pos[idx[prims, 1]])
        found.append(_hits(c, rays))
    for t, prim in found[1:]:
        np.testing.assert_array_equal(t, found[0][0])
        np.testing.assert_array_equal(prim, found[0][1])
    assert (found[0][1] >= 0).any() or kind == "flat" or n < 64
    c.close()
