"""The ray count of next-event estimation: every bounce traces one shadow ray and
one extension ray."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,spp,depth", [((64, 40), 3, 5), ((37, 23), 1, 0), ((9, 1), 2, 1), ((130, 9), 4, 9)])
@pytest.mark.parametrize("leaf", [1, 3])
def test_shadow_rays_are_counted_once(small, size, spp, depth, leaf):
    import prt
    mesh, view = small
    w, h = size
    c = prt.Context(0)
    c.load_mesh(mesh.indices, mesh.positions)
    c.set_leaf_size(leaf)
    c.build()
    c.set_integrator("diffuse2")
    c.init_frame(w, h)
    c.set_view(view, w, h)
    _, rays = c.render_profile(spp, depth)   # camera and extension rays per depth
    c.clear()
    assert c.render(spp, depth)["ray"] == rays.sum() + rays[1:].sum()
    c.close()
