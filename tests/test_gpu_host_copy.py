"""Large copies from and to pageable memory go through pinned slots filled by
several threads: the bytes equal those of a device-side or pinned copy, below
and above the sizes at which the slots are used, with ragged ends, from several
threads at once and after a context has gone."""

import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _frame(w, h):
    import prt
    import scenes
    mesh, view = scenes.small_scene()
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    c.init_frame(w, h)
    c.set_view(view, w, h)
    c.render(1, 1)
    return c


@pytest.mark.parametrize("w,h", [(61, 7), (512, 511), (513, 513), (1449, 1449), (2011, 1327)])
def test_read_accum_to_pageable_memory(w, h):
    c = _frame(w, h)
    ref = torch.empty((h, w, 4), device="cuda")
    c.read_accum(ref)
    for _ in range(2):
        np.testing.assert_array_equal(c.read_accum(), ref.cpu().numpy())
    c.close()


def test_mesh_build_from_pageable_and_pinned_memory():
    import prt
    rng = np.random.default_rng(4)
    n = 400003   # 40 MB
    soup = np.zeros(n, prt.SOUP_DTYPE)
    soup["v"]["pos"] = rng.integers(0, 60, (n, 3, 3))   # many shared vertices
    soup["v"]["normal"] = rng.normal(size=(n, 3, 3))
    soup["v"]["normal"][::2] = 0
    pinned = torch.empty(soup.nbytes, dtype=torch.uint8).pin_memory()
    pinned.copy_(torch.from_numpy(soup.view(np.uint8).reshape(-1)))
    found = []
    for src in (soup, pinned.numpy().view(prt.SOUP_DTYPE)):
        c = prt.Context(0)
        c.build_mesh(src, ["a"])
        found.append(c.read_built_mesh())
        c.close()
    for k, v in found[0].items():
        assert (v is None) == (found[1][k] is None)
        if v is not None:
            np.testing.assert_array_equal(v, found[1][k])


def test_two_threads():
    ctxs = [_frame(1449, 1449) for _ in range(2)]
    refs = [c.read_accum() for c in ctxs]
    bad = []

    def work(i):
        for _ in range(5):
            if not np.array_equal(ctxs[i].read_accum(), refs[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for c in ctxs:
        c.close()
