"""The adjoint's gradients do not depend on the workspace its chunks get: a
context without an arena cap (one chunk, packed gradient sums) against one with
a cap (a 64 KB block: many chunks, sums in the caller's arrays)."""
import numpy as np
import pytest

from umbreon_gb300 import scenes
from umbreon_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(ao=0), dict(ao=1, falloff=0.0), dict(ao=33), dict(gamma=1.8, ss=2),
                                dict(interior=True), dict(lights=0)])
@pytest.mark.parametrize("size", [(1, 1), (61, 43)])
def test_same_gradients_in_any_workspace(size, kw):
    sc, opt = scenes.differentiable(n=400, res=size[0], ao_samples=kw.get("ao", 8))
    opt.height = size[1]
    opt.supersample = kw.get("ss", 1)
    opt.aoFalloffPower = kw.get("falloff", 1.0)
    sc.assumedGamma = kw.get("gamma", 1.0)
    if "lights" in kw:
        sc.lights = sc.lights[:kw["lights"]]
    d = np.random.default_rng(2).normal(size=(size[1], size[0], 4)).astype(np.float32)
    d[::7] = 0.0
    out = []
    for cap in (0, 1 << 33):
        ctx = Context(0, arena_bytes=cap)
        b = ctx.build(sc)
        out.append(ctx.adjoint(b, sc, opt, d, interior_only=kw.get("interior", False)))
        b.release()
        ctx.close()
    a, c = out
    assert a["stats"]["samples"] == c["stats"]["samples"]
    for k in a:
        if k == "stats":
            continue
        x, y = np.asarray(a[k], np.float64), np.asarray(c[k], np.float64)
        # float sums of the same terms in another order: a sphere collects at
        # most (pixels x rays) terms, in practice a few thousand
        scale = max(np.abs(x).max(initial=0.0), 1e-30)
        assert np.abs(x - y).max(initial=0.0) <= 2e-4 * scale, k
