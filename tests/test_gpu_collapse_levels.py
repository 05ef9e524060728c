"""The 8-wide collapse at sizes around its groups of eight lanes and levels:
the default tree, the greedy one and the one with several primitives per leaf
show the same picture, for clouds and for a chain that a level only shortens."""
import numpy as np
import pytest

from umbreon_gb300 import abi
from umbreon_gb300.api import Camera, Context, DistantLight, RenderOptions, Scene

pytestmark = pytest.mark.gpu


def spheres(kind, n):
    r = np.random.default_rng(n)
    cr = np.zeros((n, 4))
    if kind == "chain":  # every split of the Morton order leaves one sphere
        cr[:, 0] = 2.0 ** -np.arange(n, dtype=np.float64)
        cr[:, 3] = 0.2 * cr[:, 0]
    elif kind == "same":  # one Morton code: the tree follows the index bits
        cr[:] = (0.5, 0.5, 0.5, 0.3)
    else:
        cr[:, :3] = r.random((n, 3))
        cr[:, 3] = 0.3 / n ** 0.4
        if kind == "outlier":  # areas above it overflow
            cr[n // 2] = (1e25, -1e25, 3e24, 1.0)
    color = np.ones((n, 4)) if kind == "same" else 0.5 + 0.5 * r.random((n, 4))
    return Scene(sphere_center_radius=cr.astype(np.float32), sphere_color=color.astype(np.float32),
                 sphere_material=np.full(n, abi.material(), abi.MATERIAL_DTYPE), lights=[DistantLight()],
                 camera=Camera(position=(0.5, 0.5, 4.0), direction=(0.0, 0.0, -1.0), orthographic=True, height=1.6))


@pytest.mark.parametrize("kind,n", [("cloud", n) for n in (1, 2, 3, 8, 9, 16, 17, 57, 129, 1025, 20000)]
                         + [("chain", 40), ("same", 300)]
                         + [("outlier", n) for n in (12, 100, 3000)])
def test_trees_show_the_same_picture(kind, n):
    sc = spheres(kind, n)
    opt = RenderOptions(width=128, height=96, aoSamples=4, aoDistance=0.5)
    pics = []
    for tree in (dict(), dict(bvh_collapse=1), dict(bvh_collapse=1, bvh_leaf_max=2), dict(bvh_collapse=2)):
        ctx = Context(0, **tree)
        built = ctx.build(sc)
        pics.append(ctx.render(built, sc, opt).color.copy())
        built.release()
        ctx.close()
    assert pics[0].any()
    for p in pics[1:]:
        assert np.array_equal(p, pics[0])
