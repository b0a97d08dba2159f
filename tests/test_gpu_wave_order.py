"""A wave takes all its passes of a pixel in turn, and camera rays of a pixel that
end together are added as one: a frame of several passes in one call equals the
sum of one-pass calls to the rounding of a pixel's sum, for passes that do and do
not divide a warp and pixels that do not fill a tile."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packets", [0, 1, 2])
@pytest.mark.parametrize("spp", [2, 3, 32, 33])
@pytest.mark.parametrize("size,depth,integrator,albedo",
                         [((37, 23), 3, "diffuse", False), ((61, 9), 0, "diffuse", True),
                          ((64, 40), 2, "diffuse", True), ((37, 23), 2, "diffuse2", True)])
def test_passes_in_one_call(small, packets, spp, size, depth, integrator, albedo):
    import prt
    import scenes
    mesh, view = small
    w, h = size
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    c.set_integrator(integrator)
    if albedo:
        c.set_albedo(scenes.albedo_for(mesh))
    c.init_frame(w, h)
    c.set_view(view, w, h)
    c.set_tune(128, 0, 0, 2, packets)
    rays = 0
    for _ in range(spp):
        rays += c.render(1, depth)["ray"]
    ref = c.read_accum()
    c.clear()
    c.set_pass(0)
    st = c.render(spp, depth)
    img = c.read_accum()
    assert st["ray"] == rays
    np.testing.assert_array_equal(img[..., 3], ref[..., 3])
    # both sums have at most two terms per ray, of at most 1 each and 2 spp in all
    terms = 2 * spp * (depth + 1)
    np.testing.assert_allclose(img[..., :3], ref[..., :3], rtol=0, atol=2.0 ** -23 * terms * 2 * spp)
    c.close()


@pytest.mark.parametrize("spp", [7, 8, 9])
def test_packets_of_large_waves(small, spp):
    """Large waves of eight passes and more take packets where no setting says
    otherwise: the same rays and sums as a launch per bounce in small waves."""
    import prt
    mesh, view = small
    w, h = 1601, 1001   # 12.9M paths in eight passes
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    c.init_frame(w, h)
    c.set_view(view, w, h)
    c.set_tune(128, 0, 1 << 24, 2, 0)
    st = c.render(spp, 2, accumulate=False)
    img = c.read_accum()
    assert c.get_tune()["primaryPackets"] == 0
    c.set_pass(0)
    c.clear()
    c.set_tune(128, 0, 2 * 1608 * 1008, 2, 0)
    _, rays = c.render_profile(spp, 2)
    ref = c.read_accum()
    assert st["ray"] == rays.sum()
    np.testing.assert_array_equal(img[..., 3], ref[..., 3])
    # up to spp terms of at most 1 on each side
    np.testing.assert_allclose(img[..., :3], ref[..., :3], rtol=0, atol=2.0 ** -23 * spp * spp)
    c.close()


def test_packets_of_large_batches(small):
    """A batch above the size that takes packets by default, in two waves that part
    inside a request, equals the requests one by one."""
    import prt
    mesh, view = small
    main = prt.Context(0)
    scene = prt.Context(0)
    scene.load_mesh(mesh.indices, mesh.positions)
    scene.build()
    shapes = [(333, 257, 21), (1001, 701, 16), (97, 5, 1)]   # 13.1M paths
    reqs = [dict(scene=scene, camera=prt.camera_from_view(view, w, h), width=w, height=h, spp=s, maxDepth=2,
                 accum=np.zeros((h, w, 4), np.float32)) for w, h, s in shapes]
    main.set_tune(128, 0, 1 << 23, 2, 0)
    st = main.render_batch(reqs)
    rays = 0
    for q in reqs:
        scene.init_frame(q["width"], q["height"])
        scene.set_view(view, q["width"], q["height"])
        scene.set_pass(0)
        rays += scene.render(q["spp"], 2, accumulate=False)["ray"]
        ref = scene.read_accum()
        np.testing.assert_array_equal(q["accum"][..., 3], ref[..., 3])
        # up to spp terms of at most 1 on each side
        np.testing.assert_allclose(q["accum"][..., :3], ref[..., :3], rtol=0, atol=2.0 ** -23 * q["spp"] ** 2)
    assert st["ray"] == rays
    scene.close()
    main.close()
