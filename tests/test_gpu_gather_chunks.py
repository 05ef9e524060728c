"""The GI gather gives the same frame whatever workspace its chunks get: a
context without an arena cap (workspace of its own, one chunk here), against
one with a cap, which gathers in the frame's hit records or, at a few pixels,
in a 64 KB block whose windows split a point's samples.  Sample counts around
the lanes per point, several bounces, emitters, adaptive refinement and ReSTIR
rounds; no lights and many lights."""
import numpy as np
import pytest

from umbreon_gb300 import scenes
from umbreon_gb300.api import Context, DistantLight

pytestmark = pytest.mark.gpu

CASES = [
    dict(pt1Spp=1), dict(pt1Spp=3, giBounces=2), dict(pt1Spp=8), dict(pt1Spp=33, giBounces=3),
    dict(pt1Spp=8, giIntegrator=1, pt1Ld=False, pt1Clamp=0.4), dict(pt1Spp=300, giIntegrator=1),
    dict(pt1Spp=9, giBounces=2, emitters=True), dict(pt1Spp=8, pt2Adaptive=True, pt2AdaptiveThresh=0.01),
    dict(pt1Spp=70, pt2Rounds=2), dict(pt1Spp=8, lights=0), dict(pt1Spp=40, lights=60),
]


@pytest.mark.parametrize("size", [(9, 7, 1), (37, 29, 2), (160, 90, 1)])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_same_frame_in_any_workspace(size, case):
    kw = dict(CASES[case])
    w, h, ss = size
    sc, opt = scenes.ball_and_stick(n=300, width=w, height=h, supersample=ss, ao_samples=0)
    if kw.pop("emitters", False):
        sc.sphere_material["emission"][::5] = 2.0
        sc.cyl_material["emission"][::7] = 1.0
    nl = kw.pop("lights", None)
    if nl is not None:
        r = np.random.default_rng(3)
        sc.lights = [DistantLight(direction=tuple(r.normal(size=3) - (0, 0, 1)), intensity=1.0 / max(nl, 1),
                                  angularRadius=0.05 * (i % 2)) for i in range(nl)]
    opt.gi, opt.giIntegrator, opt.shadows = True, 2, False
    for k, v in kw.items():
        setattr(opt, k, v)
    frames = []
    for cap in (0, 1 << 33):
        ctx = Context(0, arena_bytes=cap)
        b = ctx.build(sc)
        frames.append(ctx.render(b, sc, opt))
        b.release()
        ctx.close()
    a, c = frames
    assert a.stats["rays_primary"] == c.stats["rays_primary"]
    assert np.isfinite(a.color).all()
    assert np.array_equal(a.color, c.color)
