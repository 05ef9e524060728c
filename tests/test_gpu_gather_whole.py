"""The GI gather of few samples runs in one kernel, that of many as a wavefront.
Objects show the same bits either way: the same frame with and without a far
wall behind them, beyond the reach of their gather rays, whose points take the
frame across the line (6 launches and more instead of 2).  Per set of kinds,
which have lines of their own, at sample counts around the lanes per point, with
bounces and emitters."""
import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import Camera, Context, DistantLight, RenderOptions, Scene

pytestmark = pytest.mark.gpu

# samples up to which one kernel runs, of points that are there and of a frame
LINES = {"s": (1 << 18, 1 << 18), "sc": (1 << 15, 1 << 16), "m": (1 << 17, 1 << 17), "msc": (1 << 17, 1 << 17)}


def _scene(kinds, wall, emit):
    r = np.random.default_rng(4)
    mat = abi.material(ambient=0.2, diffuse=0.7, emission=2.0 if emit else 0.0)
    plain = abi.material(ambient=0.2, diffuse=0.7)
    sc = Scene(lights=[DistantLight(direction=(0.2, -0.3, -1.0)), DistantLight(direction=(-0.5, 0.1, -1.0))],
               camera=Camera(position=(0.0, 0.0, 60.0), direction=(0.0, 0.0, -1.0), orthographic=True, height=34.0))
    if "s" in kinds:
        n = 40
        cr = np.concatenate([r.normal(size=(n, 3)) * 1.6, r.uniform(0.4, 0.9, (n, 1))], 1)
        col = 0.4 + 0.6 * r.random((n, 4))
        mats = np.full(n, plain, abi.MATERIAL_DTYPE)
        mats[::5] = mat
        if wall and "m" not in kinds:
            cr = np.concatenate([cr, [[0.0, 0.0, -5060.0, 5000.0]]])
            col = np.concatenate([col, [[1.0, 1.0, 1.0, 1.0]]])
            mats = np.append(mats, plain)
        col[:, 3] = 1.0
        sc.sphere_center_radius, sc.sphere_color, sc.sphere_material = cr.astype(np.float32), col.astype(np.float32), mats
    if "c" in kinds:
        n = 30
        a = r.normal(size=(n, 3)) * 1.6
        sc.cyl_p0, sc.cyl_p1 = a.astype(np.float32), (a + r.normal(size=(n, 3))).astype(np.float32)
        sc.cyl_radius = np.full(n, 0.2, np.float32)
        sc.cyl_color = np.concatenate([r.random((n, 3)), np.ones((n, 1))], 1).astype(np.float32)
        sc.cyl_material = np.full(n, plain, abi.MATERIAL_DTYPE)
        sc.cyl_open = np.zeros(n, np.uint8)
    if "m" in kinds:
        m, _ = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=0, grid=1.0, width=64, height=64)
        pos = m.mesh_positions - m.mesh_positions.mean(0)
        idx = np.asarray(m.mesh_index, np.uint32).reshape(-1, 3)
        nrm, col = m.mesh_normals, m.mesh_colors.copy()
        col[:, 3] = 1.0
        if wall:
            v = len(pos)
            pos = np.concatenate([pos, [[-90, -90, -60], [90, -90, -60], [90, 90, -60], [-90, 90, -60]]])
            nrm = np.concatenate([nrm, [[0, 0, 1]] * 4])
            col = np.concatenate([col, [[1, 1, 1, 1]] * 4])
            idx = np.concatenate([idx, [[v, v + 1, v + 2], [v, v + 2, v + 3]]])
        sc.mesh_positions, sc.mesh_normals, sc.mesh_colors = pos.astype(np.float32), nrm.astype(np.float32), col.astype(np.float32)
        sc.mesh_index, sc.mesh_material = idx.astype(np.uint32), plain
    return sc


@pytest.mark.parametrize("kinds", sorted(LINES))
@pytest.mark.parametrize("spp,bounces,integrator,emit", [(1, 1, 2, False), (2, 1, 2, False), (3, 2, 1, False),
                                                         (7, 1, 2, True), (8, 1, 1, False), (8, 4, 2, False),
                                                         (8, 2, 2, True)])
def test_same_bits_on_both_sides(kinds, spp, bounces, integrator, emit):
    line, frame = (x * (2 if bounces > 2 else 1) for x in LINES[kinds])
    # a few points more than the frame's line
    h = int((frame / spp * 0.7) ** 0.5) | 1
    w = int(frame / spp / h) + 2
    opt = RenderOptions(width=w, height=h, gi=True, giIntegrator=integrator, pt1Spp=spp, giBounces=bounces,
                        giMaxDistance=20.0, pt1GatherDiv=1, pt1Denoise=False, pt1EdgePatch=False, pt2Reflect=False,
                        pt2Glossy=False)
    frames = []
    for wall in (False, True):
        sc = _scene(kinds, wall, emit)
        ctx = Context(0)
        b = ctx.build(sc)
        frames.append(ctx.render(b, sc, opt))
        b.release()
        ctx.close()
    alone, walled = frames
    there = alone.hit_geom != 0xFFFFFFFF
    assert 1000 < there.sum() * spp <= line and w * h * spp > frame
    assert np.isfinite(walled.viewZ).all() and (walled.hit_geom != 0xFFFFFFFF).all()
    assert walled.stats["kernels"] >= alone.stats["kernels"] + 4  # first, vertex, shadow, resolve, sum instead of one
    color = alone.color.reshape(h, w, 4)
    assert len(np.unique(color[there.reshape(h, w)], axis=0)) > 100
    assert np.array_equal(color[there.reshape(h, w)], walled.color.reshape(h, w, 4)[there.reshape(h, w)])
