"""A scene of triangles alone takes about the time of the same triangles with a
sphere beside them, for every kind of ray that reports its hit, and shows the
same picture."""
import copy
import ctypes as C
import time

import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import Context, make_render_desc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _scenes():
    sc, opt = scenes.molecular_surface(n_atoms=200, box=60.0 * 0.02 ** (1 / 3), n_spheres=0, width=640, height=480,
                                       ao_samples=8)
    sc.mesh_colors[:, 3] = 1.0
    both = copy.copy(sc)  # the sphere lies behind the surface, far from it
    lo, hi = sc.mesh_positions.min(0), sc.mesh_positions.max(0)
    cam = np.asarray(sc.camera.direction, np.float64)
    at = 0.5 * (lo + hi) + 50.0 * np.linalg.norm(hi - lo) * cam / np.linalg.norm(cam)
    at += 50.0 * np.linalg.norm(hi - lo) * np.cross(cam, [0.31, 0.52, 0.71])
    both.sphere_center_radius = np.array([[*at, 0.01]], np.float32)
    both.sphere_color = np.ones((1, 4), np.float32)
    both.sphere_material = np.full(1, abi.material(), abi.MATERIAL_DTYPE)
    return sc, both, opt


@pytest.mark.parametrize("kw", [dict(aoSamples=0, shadows=False), dict(aoSamples=8, aoFalloffPower=1.0),
                                dict(gi=True, giIntegrator=2, aoSamples=0, shadows=False)])
def test_frames(kw):
    sc, both, opt = _scenes()
    for k, v in kw.items():
        setattr(opt, k, v)
    ctx = Context(0)
    ms, pics = [], []
    for s in (sc, both):
        b = ctx.build(s)
        desc, keep = make_render_desc(s, opt)
        color = torch.empty((opt.height, opt.width, 4), device="cuda")
        fr = abi.Frame()
        fr.memory = abi.MEMORY_DEVICE
        fr.color = C.cast(C.c_void_p(color.data_ptr()), abi.f32p)
        t = []
        for _ in range(10):
            ctx._check(ctx._L.ubr_render(ctx.handle, b.handle, C.byref(desc), C.byref(fr), None, None))
            t.append(fr.render_ms)
        ms.append(min(t))
        pics.append(color.cpu().numpy())
        b.release()
    ctx.close()
    assert np.array_equal(*pics)
    assert ms[0] < 1.3 * ms[1], ms


def test_filtered_segments():
    sc, both, _ = _scenes()
    n = 200000
    r = np.random.default_rng(1)
    lo, hi = sc.mesh_positions.min(0), sc.mesh_positions.max(0)
    segs = torch.from_numpy((lo + r.random((n, 2, 3)) * (hi - lo)).reshape(n, 6).astype(np.float32)).cuda()
    ctx = Context(0)
    ms, got = [], []
    for s in (sc, both):
        b = ctx.build(s)
        out = torch.empty(n, dtype=torch.uint8, device="cuda")
        t = []
        for _ in range(10):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            ctx._check(ctx._L.ubr_occluded_filtered_batch(ctx.handle, b.handle, segs.data_ptr(), n, 1e-4, 1e-3, 0.0,
                                                          None, None, out.data_ptr(), abi.MEMORY_DEVICE))
            t.append(time.perf_counter() - t0)
        ms.append(min(t))
        got.append(out.cpu().numpy())
        b.release()
    ctx.close()
    assert np.array_equal(*got)
    assert ms[0] < 1.3 * ms[1], ms
