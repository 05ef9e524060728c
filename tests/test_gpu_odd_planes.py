"""Device planes at addresses that are no multiple of their element (a copy takes
them, a kernel's store would not): the same planes as in host buffers."""
import ctypes as C

import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import AOV_FIELDS, Context, make_render_desc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shift", [1, 2, 3, 4, 7, 12])
def test_planes_at_odd_addresses(shift):
    sc, opt = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=30, grid=1.0, width=67, height=41, ao_samples=4)
    opt.aoWriteAov = True
    ctx = Context(0)
    b = ctx.build(sc)
    want = ctx.render(b, sc, opt)
    host = dict(color=want.color, depth=want.depth, view_z=want.viewZ, hit_geom=want.hit_geom, hit_prim=want.hit_prim,
                **{c: getattr(want, n) for n, c, _ in AOV_FIELDS})
    desc, keep = make_render_desc(sc, opt)
    fr = abi.Frame()
    fr.memory = abi.MEMORY_DEVICE
    bufs = {}
    for name, w in host.items():
        t = torch.full((w.nbytes + 16,), 7, dtype=torch.uint8, device="cuda")
        bufs[name] = t
        setattr(fr, name, C.cast(C.c_void_p(t.data_ptr() + shift), abi.u32p if name.startswith("hit") else abi.f32p))
    ctx._check(ctx._L.ubr_render(ctx.handle, b.handle, C.byref(desc), C.byref(fr), None, None))
    for name, w in host.items():
        got = bufs[name].cpu().numpy()
        assert (got[:shift] == 7).all() and (got[shift + w.nbytes:] == 7).all(), name
        assert got[shift:shift + w.nbytes].tobytes() == np.ascontiguousarray(w).tobytes(), name
    b.release()
    ctx.close()
