"""The adjoint's per-sphere arrays in the caller's memory: device memory gets the
packed sums spread over it at the end; memory that the device does not hold as
its own (here page-locked host memory, which kernels can reach) is cleared and
added to.  Same gradients as in host arrays, some arrays left out."""
import ctypes as C

import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.api import Context, make_render_desc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("skip", [(), ("sphere_center",), ("sphere_color", "sphere_radius")])
@pytest.mark.parametrize("where", ["device", "pinned", "both"])
def test_per_sphere_arrays(where, skip):
    sc, opt = scenes.differentiable(n=300, res=48, ao_samples=4)
    n = sc.sphere_count()
    d = np.random.default_rng(3).normal(size=(opt.height, opt.width, 4)).astype(np.float32)
    ctx = Context(0)
    b = ctx.build(sc)
    want = ctx.adjoint(b, sc, opt, d)
    desc, keep = make_render_desc(sc, opt)
    dc = torch.from_numpy(d).cuda()
    torch.cuda.synchronize()
    g = abi.Grads()
    g.memory = abi.MEMORY_DEVICE
    bufs = {}
    for k, (name, ch) in enumerate((("sphere_color", 3), ("sphere_center", 3), ("sphere_radius", 1))):
        pinned = where == "pinned" or (where == "both" and k == 1)
        t = torch.full((n * ch,), 9.0).pin_memory() if pinned else torch.full((n * ch,), 9.0, device="cuda")
        torch.cuda.synchronize()
        bufs[name] = t
        if name not in skip:
            setattr(g, name, C.cast(C.c_void_p(t.data_ptr()), abi.f32p))
    ctx._check(ctx._L.ubr_adjoint(ctx.handle, b.handle, C.byref(desc), dc.data_ptr(), C.byref(g)))
    for name, t in bufs.items():
        got = t.cpu().numpy()
        if name in skip:
            assert (got == 9.0).all(), name
        else:
            w = np.asarray(want[name]).reshape(-1)
            # float sums of the same terms in another order
            assert np.abs(got - w).max() <= 2e-4 * max(np.abs(w).max(), 1e-30), name
    b.release()
    ctx.close()
