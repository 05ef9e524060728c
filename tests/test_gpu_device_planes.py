"""Frames into device buffers: the planes written in place equal the ones copied
to host buffers, for every kind of frame that is written in place or is not
(grid, transparent layers, AOVs and denoiser, GI, adaptive AA, edge G-buffer,
batch), with planes left out, a colour buffer that is not 16-byte aligned, and
other buffers in the next call (a captured graph keeps no pointer of a call)."""
import ctypes as C

import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import AOV_FIELDS, Context, make_render_desc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PLANES = ("color", "depth", "view_z", "hit_geom", "hit_prim")


def _cases(name):
    if name in ("surface", "surface_aov", "edge"):
        sc, opt = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=30, grid=1.0, width=67, height=41,
                                           ao_samples=4)
        if name == "surface_aov":
            sc.mesh_colors[:, 3] = 1.0
            opt.aoWriteAov, opt.aoFalloffPower, opt.denoiser = True, 1.0, 1
        opt.edgeGBuffer = name == "edge"
        return sc, opt
    sc, opt = scenes.ball_and_stick(n=200, width=67, height=41, supersample=1 if name == "grid" else 2, ao_samples=4)
    opt.gi = name == "gi"
    opt.aaMode = 1 if name == "adaptive" else 0
    return sc, opt


def _frame(opt, skip=(), shift=0):
    ss = max(1, opt.supersample)
    fr = abi.Frame()
    fr.memory = abi.MEMORY_DEVICE
    bufs = {}
    for name in PLANES + tuple(a[1] for a in AOV_FIELDS if opt.aoWriteAov):
        ch = dict(color=4, **{a[1]: a[2] for a in AOV_FIELDS}).get(name, 1)
        px = opt.width * opt.height * (1 if name == "color" or name not in PLANES else ss * ss)
        t = torch.full((px * ch + shift,), -7.0, device="cuda")
        bufs[name] = t[shift:]
        if name not in skip:
            setattr(fr, name, C.cast(C.c_void_p(t.data_ptr() + 4 * shift),
                                     abi.u32p if name.startswith("hit") else abi.f32p))
    return fr, bufs


def _check(bufs, want, skip=()):
    host = dict(color=want.color, depth=want.depth, view_z=want.viewZ, hit_geom=want.hit_geom, hit_prim=want.hit_prim,
                **{c: getattr(want, n) for n, c, _ in AOV_FIELDS})
    for name, t in bufs.items():
        got = t.cpu().numpy()
        if name in skip:
            assert (got == -7.0).all(), name
        else:
            w = np.ascontiguousarray(host[name]).reshape(-1).view(np.float32)
            assert np.array_equal(got.view(np.uint32), w.view(np.uint32)), name


@pytest.mark.parametrize("name", ["grid", "surface", "surface_aov", "edge", "gi", "adaptive", "ss2"])
def test_planes_in_device_buffers(name):
    sc, opt = _cases(name)
    ctx = Context(0)
    b = ctx.build(sc)
    want = ctx.render(b, sc, opt)
    desc, keep = make_render_desc(sc, opt)
    for skip, shift in (((), 0), ((), 0), (("depth", "hit_prim"), 0), (("view_z",), 1), (("color",), 0)):
        fr, bufs = _frame(opt, skip, shift)
        ctx._check(ctx._L.ubr_render(ctx.handle, b.handle, C.byref(desc), C.byref(fr), None, None))
        _check(bufs, want, skip)
    b.release()
    ctx.close()


def test_batch_into_device_buffers():
    ctx = Context(0)
    items = [_cases(n) for n in ("grid", "surface_aov", "surface", "ss2", "adaptive")]
    items[1][1].denoiser = 0
    built = [ctx.build(sc) for sc, _ in items]
    want = [ctx.render(b, sc, opt) for b, (sc, opt) in zip(built, items)]
    arr = (abi.BatchItem * len(items))()
    frames = [_frame(opt, skip=("hit_geom",) if i == 2 else ()) for i, (_, opt) in enumerate(items)]
    keep = []
    for i, (b, (sc, opt)) in enumerate(zip(built, items)):
        desc, k = make_render_desc(sc, opt)
        keep += [desc, k]
        arr[i].scene, arr[i].desc, arr[i].frame = b.handle, C.pointer(desc), C.pointer(frames[i][0])
    for _ in range(2):
        ctx._check(ctx._L.ubr_render_batch(ctx.handle, len(items), arr, None))
    for i, ((fr, bufs), w) in enumerate(zip(frames, want)):
        _check(bufs, w, ("hit_geom",) if i == 2 else ())
    for b in built:
        b.release()
    ctx.close()
