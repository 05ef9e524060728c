"""Segment queries per set of primitive kinds: spheres, spheres + bonds, a mesh,
mesh + spheres, everything (round cylinders too), at segment counts around the
block size, against the oracle's any-hit test; the allocation-free query and
the filtered query without filters give the same bytes."""
import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import Scene

pytestmark = pytest.mark.gpu


def _scene(kinds):
    sc, _ = scenes.ball_and_stick(n=300, width=64, height=64, supersample=1, ao_samples=0)
    if "round" in kinds:
        sc.cyl_open = (np.arange(len(sc.cyl_p0)) % 2).astype(np.uint8)
    if "cone" not in kinds:
        sc.cyl_p0 = sc.cyl_p1 = sc.cyl_radius = sc.cyl_color = sc.cyl_material = sc.cyl_open = None
    if "mesh" in kinds:
        m, _ = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=0, grid=1.0, width=64, height=64)
        sc.mesh_positions = m.mesh_positions + sc.sphere_center_radius[:, :3].mean(0) - 6.0
        sc.mesh_normals, sc.mesh_colors, sc.mesh_index = m.mesh_normals, m.mesh_colors, m.mesh_index
        sc.mesh_material = m.mesh_material
    if "sphere" not in kinds:
        sc.sphere_center_radius = sc.sphere_color = sc.sphere_material = None
    return sc


@pytest.mark.parametrize("kinds", [("sphere",), ("sphere", "cone"), ("mesh",), ("mesh", "sphere"),
                                   ("sphere", "cone", "round", "mesh")])
@pytest.mark.parametrize("n", [1, 127, 129, 20000])
def test_segments(gpu_ctx, oracle_lib, kinds, n):
    sc = _scene(kinds)
    r = np.random.default_rng(n)
    pts = sc.mesh_positions if "mesh" in kinds else sc.sphere_center_radius[:, :3]
    lo, hi = pts.min(0) - 2.0, pts.max(0) + 2.0
    segs = np.concatenate([lo + r.random((n, 3)) * (hi - lo), lo + r.random((n, 3)) * (hi - lo)], 1).astype(np.float32)
    b = gpu_ctx.build(sc)
    got = gpu_ctx.occluded(b, segs, 1e-4)
    same = gpu_ctx.occluded_filtered(b, segs, 1e-4)
    out = np.zeros(n, np.uint8)
    st = gpu_ctx._L.ubr_occluded_batch_noalloc(gpu_ctx.handle, b.handle, segs.ctypes.data, n, 1e-4, out.ctypes.data)
    b.release()
    assert st == abi.UBR_OK
    assert np.array_equal(got, same) and np.array_equal(got, out)
    want = oracle_lib.OracleScene(sc).occluded_filtered(segs, 1e-4)
    # a segment that grazes a surface may answer differently; the queries above
    # the block size meet a few, the small ones none
    assert np.mean(got != want) <= 5e-4
