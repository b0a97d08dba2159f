"""prt_render_noalloc over several waves.  With packets each wave of a frame that
fills the fixed array is one pass, so that its queue and throughputs are filled and
used again; without a queue a wave ends only at 2^30 items."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packets", [0, 1, 2])
@pytest.mark.parametrize("albedo", [False, True])
@pytest.mark.parametrize("w,h", [(1024, 512), (1021, 509)])
def test_noalloc_waves_equal_render(small, packets, albedo, w, h):
    import prt
    import scenes
    mesh, view = small
    spp, depth = 3, 5
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    if albedo:
        c.set_albedo(scenes.albedo_for(mesh))
    c.build()
    c.init_frame(w, h)
    cam = prt.camera_from_view(view, w, h)
    c.set_camera(cam)
    c.set_tune(128, 0, 0, 2, packets)
    c.set_pass(2)
    st = c.render(spp, depth, accumulate=False)
    ref = c.read_accum()
    for _ in range(2):   # the second call meets the array the first left behind
        acc = torch.zeros((h, w, 4), device="cuda")
        torch.cuda.synchronize()
        rays = c.render_noalloc(cam, w, h, 2, spp, depth, acc)
        img = acc.cpu().numpy()
        assert rays == st["ray"]
        np.testing.assert_array_equal(img[..., 3], ref[..., 3])
        # up to spp terms of at most 1 on each side
        np.testing.assert_allclose(img[..., :3], ref[..., :3], rtol=0, atol=2.0 ** -23 * spp * spp)
    c.close()


@pytest.mark.parametrize("integrator", ["diffuse", "diffuse2"])
def test_waves_of_many_passes(integrator):
    """2049 passes of 524288 pixels of sky: 2^30 + 2^19 items, so two waves."""
    import prt
    import scenes
    w, h, spp = 1024, 512, 2049
    c = prt.Context(0)
    c.load_mesh(np.zeros((0, 3), np.int32), np.zeros((0, 3), np.float32))
    c.build()
    c.set_integrator(integrator)
    cam = prt.camera_from_view(scenes.View((0.0, 0.0, 5.0), 0.0, 0.0, 0.7, 0.0, 5.0), w, h)
    acc = torch.zeros((h, w, 4), device="cuda")
    torch.cuda.synchronize()
    assert c.render_noalloc(cam, w, h, 0, spp, 2, acc) == w * h * spp
    # every path adds 1: whole numbers, exact
    assert bool((acc == spp).all())
    c.close()
