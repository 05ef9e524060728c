"""Device planes that overlap: frames of a batch that share a plane nobody reads
(view z, depth, ids as throw-aways), and planes of one frame that share memory.
Every other plane is what it is with buffers of its own."""
import copy
import ctypes as C

import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import Context, Fog, make_render_desc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PLANES = ("color", "depth", "view_z", "hit_geom", "hit_prim")
TYPES = dict(color=abi.f32p, depth=abi.f32p, view_z=abi.f32p, hit_geom=abi.u32p, hit_prim=abi.u32p)


def _scene(k):
    """Transparent surface (several layers) with fog, another view per k."""
    sc, opt = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=30, grid=1.0, width=61 + 6 * k, height=41,
                                       ao_samples=4)
    sc.fog = Fog(enabled=True, color=(0.9, 0.8, 0.7), start=5.0, end=60.0)
    return sc, opt


def _want(frame, name):
    host = dict(color=frame.color, depth=frame.depth, view_z=frame.viewZ, hit_geom=frame.hit_geom,
                hit_prim=frame.hit_prim)
    return np.ascontiguousarray(host[name]).reshape(-1).view(np.uint32)


def _buf(opt, name):
    return torch.full((opt.width * opt.height * (4 if name == "color" else 1),), -7.0, device="cuda")


def _set(fr, name, t, at=0):
    setattr(fr, name, C.cast(C.c_void_p(t.data_ptr() + at), TYPES[name]))


@pytest.mark.parametrize("shared", [("view_z",), ("depth",), ("depth", "view_z", "hit_geom", "hit_prim")])
def test_batch_frames_share_a_plane(shared):
    ctx = Context(0)
    items = [_scene(k) for k in range(3)]
    built = [ctx.build(sc) for sc, _ in items]
    want = [ctx.render(b, sc, opt) for b, (sc, opt) in zip(built, items)]
    common = {n: _buf(items[-1][1], n) for n in shared}
    arr = (abi.BatchItem * 3)()
    keep, bufs = [], []
    for i, (b, (sc, opt)) in enumerate(zip(built, items)):
        desc, k = make_render_desc(sc, opt)
        fr = abi.Frame()
        fr.memory = abi.MEMORY_DEVICE
        own = {n: common[n] if n in shared else _buf(opt, n) for n in PLANES}
        for n, t in own.items():
            _set(fr, n, t)
        arr[i].scene, arr[i].desc, arr[i].frame = b.handle, C.pointer(desc), C.pointer(fr)
        keep += [desc, k, fr]
        bufs.append(own)
    ctx._check(ctx._L.ubr_render_batch(ctx.handle, 3, arr, None))
    for own, w in zip(bufs, want):
        for n in PLANES:
            if n not in shared:
                assert np.array_equal(own[n].cpu().numpy().view(np.uint32), _want(w, n)), n
    for b in built:
        b.release()
    ctx.close()


@pytest.mark.parametrize("pair", [("view_z", "hit_prim"), ("depth", "hit_geom"), ("depth", "view_z")])
def test_planes_of_a_frame_share_memory(pair):
    """The later plane of the pair (colour, depth, view z, ids in this order) is
    the one left in the shared buffer, and the others are untouched by it."""
    ctx = Context(0)
    sc, opt = _scene(0)
    b = ctx.build(sc)
    want = ctx.render(b, sc, opt)
    desc, keep = make_render_desc(sc, opt)
    fr = abi.Frame()
    fr.memory = abi.MEMORY_DEVICE
    bufs = {n: _buf(opt, n) for n in PLANES}
    bufs[pair[0]] = bufs[pair[1]]
    for n in PLANES:
        _set(fr, n, bufs[n])
    ctx._check(ctx._L.ubr_render(ctx.handle, b.handle, C.byref(desc), C.byref(fr), None, None))
    for n in PLANES:
        if n != pair[0]:
            assert np.array_equal(bufs[n].cpu().numpy().view(np.uint32), _want(want, n)), n
    b.release()
    ctx.close()
