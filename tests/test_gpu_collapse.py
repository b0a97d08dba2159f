"""The collapse into 8-wide nodes: warps with one to four nodes, leaves of one to
three triangles, both groupings, trees of more levels than are launched before
the counters are first read; and sorts whose digit rows take several steps.
Every triangle is in one leaf and closest hits do not depend on the tree."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _soup(n, deep, seed=3):
    rng = np.random.default_rng(seed + n)
    c = rng.uniform(-1, 1, (n, 1, 3))
    size = np.full((n, 1, 1), 0.5 * n ** -0.4)
    if deep:
        # each triangle twice as far out and as large as the one before
        size = 2.0 ** (np.arange(n).reshape(-1, 1, 1) * 0.5 - 0.25 * n)
        c = np.ones((n, 1, 3)) * size * 4
    return (c + rng.uniform(-1, 1, (n, 3, 3)) * size).astype(np.float32).reshape(-1, 3), \
        np.arange(3 * n, dtype=np.int32).reshape(n, 3)


@pytest.mark.parametrize("n, deep", [(1, False), (2, False), (9, False), (33, False), (700, False), (120, True)])
def test_collapse(n, deep):
    import prt
    pos, idx = _soup(n, deep)
    g = torch.Generator(device="cuda").manual_seed(n)
    m = 2048
    rays = torch.zeros((m, 8), device="cuda")
    target = torch.from_numpy(pos.reshape(n, 3, 3).mean(1)).cuda()
    target = target[torch.randint(0, n, (m,), generator=g, device="cuda")]
    rays[:, :3] = torch.randn((m, 3), generator=g, device="cuda")
    d = target - rays[:, :3]
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1e30
    hits = torch.empty((m, 4), device="cuda")
    torch.cuda.synchronize()
    c = prt.Context(0)
    c.load_mesh(idx, pos)
    want = None
    for high in (True, False):
        for leaf in (1, 2, 3):
            c.set_build_quality(high)
            c.set_leaf_size(leaf)
            info = c.build()
            nodes, tris = c.read_accel()
            prims = tris[:, 3].view(np.int32)
            np.testing.assert_array_equal(np.sort(prims), np.arange(n))
            np.testing.assert_array_equal(tris[:, 4:7], pos[idx[prims, 1]])
            assert info["nodeCount"] == len(nodes)
            if deep and high:
                assert info["levels"] > 4   # launched before the first read-back
            c.intersect(rays, hits, m)
            torch.cuda.synchronize()
            got = hits[:, :2].cpu().numpy().copy().view(np.int32)
            assert (got[:, 1] >= 0).any()
            if deep:
                continue   # most triangles are smaller than an ulp of their distance: any of them is the hit
            want = got if want is None else want
            np.testing.assert_array_equal(got, want)
    c.close()


def test_sort_of_many_tiles():
    import prt
    n = 257 * 4096 + 5   # more tiles than a digit's row takes in one step
    pos, idx = _soup(n, False)
    c = prt.Context(0)
    c.load_mesh(idx, pos)
    c.set_build_quality(False)   # the Morton tree needs sorted keys
    c.build()
    _, tris = c.read_accel()
    np.testing.assert_array_equal(np.sort(tris[:, 3].view(np.int32)), np.arange(n))
    rays = torch.zeros((4096, 8), device="cuda")
    rays[:, :3] = torch.rand((4096, 3), device="cuda") * 2 - 1
    rays[:, 4:7] = torch.nn.functional.normalize(torch.randn((4096, 3), device="cuda"), dim=1)
    rays[:, 7] = 1e30
    found = []
    for high in (False, True):
        c.set_build_quality(high)
        c.build()
        hits = torch.empty((4096, 4), device="cuda")
        torch.cuda.synchronize()
        c.intersect(rays, hits, 4096)
        torch.cuda.synchronize()
        found.append(hits[:, :2].cpu().numpy().copy().view(np.int32))
    np.testing.assert_array_equal(found[0], found[1])
    c.close()
