"""prt_render carries paths through all bounces in one launch, which starts with
the camera rays for small waves and next-event estimation and takes a queue of
paths otherwise; prt_render_profile does one launch per bounce.  Both trace the same paths, so their frames agree to
the rounding of a pixel's sum (at most spp additions of values up to 1) and
their ray counts are equal."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["diffuse", "diffuse2"])
@pytest.mark.parametrize("albedo", [False, True])
@pytest.mark.parametrize("leaf,size,depth", [(1, (64, 40), 5), (1, (37, 23), 0), (1, (9, 1), 1), (1, (130, 9), 9),
                                             (2, (37, 23), 3), (3, (64, 40), 2)])
def test_whole_paths_equal_bounce_by_bounce(small, integrator, albedo, leaf, size, depth):
    import prt
    import scenes
    mesh, view = small
    w, h = size
    spp = 3
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.set_leaf_size(leaf)
    c.build()
    c.set_integrator(integrator)
    if albedo:
        c.set_albedo(scenes.albedo_for(mesh))
    c.init_frame(w, h)
    c.set_view(view, w, h)
    _, rays = c.render_profile(spp, depth)
    ref = c.read_accum()
    c.clear()
    st = c.render(spp, depth)
    img = c.read_accum()
    np.testing.assert_array_equal(img[..., 3], ref[..., 3])
    # each sum of up to spp terms (two per bounce with shadow rays) of at most 1 rounds by 2^-24 a term
    np.testing.assert_allclose(img[..., :3], ref[..., :3], rtol=0, atol=2.0 ** -24 * spp * spp)
    if integrator == "diffuse":
        assert st["ray"] == rays.sum()   # render_profile counts queue entries, not shadow rays
    else:
        assert st["ray"] >= rays.sum()
    c.close()


@pytest.mark.parametrize("packets", [0, 1, 2])
@pytest.mark.parametrize("albedo", [False, True])
@pytest.mark.parametrize("waves", [1, 3])
def test_queued_paths_equal_bounce_by_bounce(small, packets, albedo, waves):
    """Waves above the size that starts in one launch (10240 paths per SM), or
    with packet primaries at any size, go through the queue."""
    import prt
    import scenes
    mesh, view = small
    w, h = (1931, 1087) if packets == 0 else (203, 101)
    spp = 3
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    if albedo:
        c.set_albedo(scenes.albedo_for(mesh))
    c.init_frame(w, h)
    c.set_view(view, w, h)
    per_pass = ((w + 7) // 8) * ((h + 7) // 8) * 64
    c.set_tune(128, 0, per_pass * (spp // waves), 2, packets)
    _, rays = c.render_profile(spp, 4)
    ref = c.read_accum()
    c.clear()
    for _ in range(2):   # the second call replays a recorded graph if there are several waves
        c.set_pass(0)
        st = c.render(spp, 4, accumulate=False)
        img = c.read_accum()
        np.testing.assert_array_equal(img[..., 3], ref[..., 3])
        np.testing.assert_allclose(img[..., :3], ref[..., :3], rtol=0, atol=2.0 ** -24 * spp * spp)
        assert st["ray"] == rays.sum() and c.get_pass() == spp
    c.close()
