"""Gather rays through spheres and cylinders put their primitive tests off;
with a triangle out of sight the same frame takes the general traversal: equal
pictures, at ray counts that leave warps partly or wholly empty and at trees
of one node, of leaves only and of several levels."""
import numpy as np
import pytest

from umbreon_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size,spp", [(1, (9, 7), 1), (2, (33, 17), 3), (5, (33, 17), 8), (40, (64, 48), 5),
                                        (700, (96, 54), 16), (5000, (160, 90), 33)])
@pytest.mark.parametrize("integrator,bounces", [(1, 1), (2, 1), (1, 3), (2, 2)])
def test_same_frame_as_the_general_traversal(gpu_ctx, n, size, spp, integrator, bounces):
    pics = []
    for far in (False, True):
        sc, opt = scenes.ball_and_stick(n=n, width=size[0], height=size[1], supersample=1, ao_samples=0)
        opt.gi, opt.giIntegrator, opt.pt1Spp, opt.giBounces, opt.shadows = True, integrator, spp, bounces, False
        if far:  # a speck behind the camera
            p = np.asarray(sc.camera.position) - 500.0 * np.asarray(sc.camera.direction)
            sc.mesh_positions = (p + 1e-5 * np.eye(3)).astype(np.float32)
        b = gpu_ctx.build(sc)
        pics.append(gpu_ctx.render(b, sc, opt))
        b.release()
    assert pics[0].stats["rays_primary"] == pics[1].stats["rays_primary"]
    assert pics[0].color.any()
    assert np.array_equal(pics[0].color, pics[1].color)
