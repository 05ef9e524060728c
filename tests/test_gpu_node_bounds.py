"""The wide nodes' quantised boxes hold at every scale, offset and flatness of
a scene, and with one or several primitives per leaf: first hits and segment
visibility of sphere clouds against brute force in float64."""
import numpy as np
import pytest

from umbreon_gb300 import abi
from umbreon_gb300.api import Camera, Context, DistantLight, RenderOptions, Scene

pytestmark = pytest.mark.gpu

TREES = [dict(), dict(bvh_leaf_max=3), dict(bvh_collapse=2), dict(bvh_builder=2, bvh_collapse=2, sah_prim_scale=4.0)]


def cloud(n, scale, offset, flat, seed):
    r = np.random.default_rng(seed)
    c = r.random((n, 3)) * np.array([1.0, 1.0, 0.0 if flat else 1.0])
    rad = 0.01 + 0.04 * r.random(n)
    cr = np.concatenate([c * scale + offset, rad[:, None] * scale], 1).astype(np.float32)
    return Scene(sphere_center_radius=cr, sphere_color=np.ones((n, 4), np.float32),
                 sphere_material=np.full(n, abi.material(), abi.MATERIAL_DTYPE),
                 lights=[DistantLight()])


@pytest.mark.parametrize("n,scale,offset,flat", [(1, 1.0, 0.0, False), (2, 1.0, 0.0, False), (9, 1.0, 0.0, True),
                                                 (300, 1e-3, 0.0, False), (300, 1.0, 40.0, True),
                                                 (2000, 1e4, 0.0, False), (2000, 1.0, -20.0, False)])
def test_hits_and_segments_match_brute_force(n, scale, offset, flat):
    sc = cloud(n, scale, offset, flat, 5 + n)
    W = H = 65
    mid = np.array([0.5, 0.5, 0.0]) * scale + offset
    sc.camera = Camera(position=tuple(mid + np.array([0.0, 0.0, 3.0 * scale])), direction=(0.0, 0.0, -1.0),
                       orthographic=True, height=1.1 * scale)
    cr = sc.sphere_center_radius.astype(np.float64)
    u = (2.0 * (np.arange(W) + 0.5) / W - 1.0) * 0.55 * scale
    x, y = mid[0] + u, mid[1] - u
    d2 = (x[None, :, None] - cr[:, 0]) ** 2 + (y[:, None, None] - cr[:, 1]) ** 2
    q = cr[:, 3] ** 2 - d2
    top = np.where(q >= 0, cr[:, 2] + np.sqrt(np.maximum(q, 0.0)), -np.inf)
    # float positions carry 2^-23 of the coordinate: a few of those per sphere
    # test, against a radius of at least 0.01 of the scale
    tol = 64.0 * 2.0 ** -23 * (abs(offset) + 4.0 * scale)
    order = np.sort(top, -1)
    graze = np.any(np.abs(np.sqrt(d2) - cr[:, 3]) < tol, -1)
    near = np.zeros((H, W), bool)
    if n > 1:
        with np.errstate(invalid="ignore"):  # background: -inf - -inf
            near = order[..., -1] - order[..., -2] < 4.0 * tol * (1.0 + scale / tol) ** 0.5
    sure = ~(graze | near)
    prim = np.where(np.isfinite(order[..., -1]), np.argmax(top, -1), 0xFFFFFFFF).astype(np.uint32)
    assert sure.mean() > 0.6

    r = np.random.default_rng(1)
    m = 4000
    a = r.random((m, 3)) * scale + offset
    b = r.random((m, 3)) * scale + offset
    if flat:
        a[:, 2], b[:, 2] = mid[2] - 0.2 * scale, mid[2] + 0.2 * scale
    segs = np.concatenate([a, b], 1).astype(np.float32)
    p0, p1 = segs[:, :3].astype(np.float64), segs[:, 3:].astype(np.float64)
    d = p1 - p0
    ln = np.linalg.norm(d, axis=1)
    rel = cr[None, :, :3] - p0[:, None, :]
    t = np.clip((rel * d[:, None, :]).sum(-1) / (ln ** 2)[:, None], 0.0, 1.0)
    dist = np.linalg.norm(rel - t[..., None] * d[:, None, :], axis=-1)
    in0 = np.linalg.norm(rel, axis=-1) < cr[:, 3] + tol
    in1 = np.linalg.norm(cr[None, :, :3] - p1[:, None, :], axis=-1) < cr[:, 3] + tol
    blocked = np.any(dist < cr[:, 3], -1)
    clear = ~(np.any(np.abs(dist - cr[:, 3]) < tol, -1) | np.any(in0 | in1, -1)) & (ln > 0.05 * scale)
    assert clear.mean() > 0.2

    for tree in TREES:
        ctx = Context(0, **tree)
        built = ctx.build(sc)
        fr = ctx.render(built, sc, RenderOptions(width=W, height=H))
        got = ctx.occluded(built, segs, 1e-6)
        built.release()
        ctx.close()
        assert np.array_equal(fr.hit_prim[sure], prim[sure]), tree
        assert np.array_equal(got[clear].astype(bool), blocked[clear]), tree
