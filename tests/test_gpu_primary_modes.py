"""Camera rays per lane on request (prt_tune.primaryPackets = 3), where the library
would choose packets: the same frame, the setting kept and reported."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_per_lane_setting(small):
    import prt
    mesh, view = small
    w, h, spp = 1601, 1001, 8   # 12.9M paths: packets without a setting
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    c.init_frame(w, h)
    c.set_view(view, w, h)
    frames = []
    for mode in (0, 3):
        c.set_tune(128, 0, 1 << 24, 2, mode)
        assert c.get_tune()["primaryPackets"] == mode
        c.set_pass(0)
        frames.append((c.render(spp, 2, accumulate=False)["ray"], c.read_accum()))
    assert frames[0][0] == frames[1][0]
    # up to spp terms of at most 1 on each side
    np.testing.assert_allclose(frames[0][1], frames[1][1], rtol=0, atol=2.0 ** -23 * spp * spp)
    for bad in (-1, 4):
        with pytest.raises(prt.PrtError) as e:
            c.set_tune(128, 0, 0, 2, bad)
        assert e.value.status == prt.PRT_EINVAL
    assert c.get_tune()["primaryPackets"] == 3

    batch = []
    for mode in (0, 3):
        c.set_tune(128, 0, 0, 2, mode)
        req = dict(scene=c, camera=prt.camera_from_view(view, w, h), width=w, height=h, spp=spp, maxDepth=2,
                   accum=np.zeros((h, w, 4), np.float32))
        batch.append((c.render_batch([req])["ray"], req["accum"]))
        assert batch[-1][0] == frames[0][0]
        np.testing.assert_allclose(batch[-1][1], frames[0][1], rtol=0, atol=2.0 ** -23 * spp * spp)
    c.close()


def test_profile_traces_camera_rays_as_the_renderer(small):
    """prt_render_profile's first bounce is the kernel prt_render takes in large
    waves: without a setting its time is that of packets, not of lanes."""
    import prt
    mesh, view = small
    w, h, spp = 1601, 1001, 8
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.build()
    c.init_frame(w, h)
    c.set_view(view, w, h)
    ms = {0: [], 1: [], 3: []}
    for _ in range(6):
        for mode in ms:
            c.set_tune(128, 0, 1 << 24, 2, mode)
            ms[mode].append(c.render_profile(spp, 2)[0][0])
    library, packets, lanes = (min(ms[m][1:]) for m in (0, 1, 3))
    assert abs(library - packets) < abs(library - lanes), ms
    c.close()
