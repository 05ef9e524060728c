"""Large launches of binary occlusion rays through spheres and cylinders run the
kernel whose warps fetch rays; the frames are those of one thread per ray
(trace_mode 1), around the launch size where the choice changes, alone, in a
batch and under adaptive AA (which copies rays of an earlier pass)."""
import numpy as np
import pytest

from umbreon_gb300 import scenes
from umbreon_gb300.api import Context

pytestmark = pytest.mark.gpu


def _scene(model, w, h, ao, ss=1):
    if model == "spheres":
        sc, opt = scenes.space_filling(n=3000, width=w, height=h)
        opt.aoSamples, opt.aoDistance, opt.shadows, opt.supersample = ao, 5.0, ao % 2 == 0, ss
    else:
        sc, opt = scenes.ball_and_stick(n=900, width=w, height=h, supersample=ss, ao_samples=ao)
    return sc, opt


def _same(a, b):
    for k in ("color", "depth", "viewZ", "hit_geom", "hit_prim"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.stats["rays_occlusion"] == b.stats["rays_occlusion"]


# 12,000,000 rays counting misses: just below, just above, and well above, odd
# sizes, ray counts per hit that are not multiples of a warp
@pytest.mark.parametrize("model,w,h,ao,ss", [
    ("spheres", 1000, 705, 16, 1), ("spheres", 1001, 707, 16, 1), ("spheres", 1283, 721, 13, 1),
    ("ball", 999, 667, 16, 1), ("ball", 1001, 667, 16, 1), ("ball", 641, 479, 37, 2), ("ball", 1400, 1000, 7, 1)])
def test_single_frames(model, w, h, ao, ss):
    sc, opt = _scene(model, w, h, ao, ss)
    out = []
    for mode in (0, 1):
        ctx = Context(0, trace_mode=mode)
        b = ctx.build(sc)
        out.append(ctx.render(b, sc, opt))
        b.release()
        ctx.close()
    _same(*out)


def test_batch_and_adaptive():
    items = [_scene(m, w, h, ao) for m, w, h, ao in (("spheres", 700, 613, 16), ("ball", 811, 600, 9),
                                                     ("spheres", 257, 255, 0), ("ball", 640, 480, 16))]
    sc_a, opt_a = _scene("ball", 901, 853, 16, 2)
    opt_a.aaMode = 1
    out = []
    for mode in (0, 1):
        ctx = Context(0, trace_mode=mode)
        built = [(ctx.build(sc), sc, opt) for sc, opt in items]
        frames, _ = ctx.render_batch(built)
        ba = ctx.build(sc_a)
        adaptive = ctx.render(ba, sc_a, opt_a)
        for b, _, _ in built:
            b.release()
        ba.release()
        ctx.close()
        out.append((frames, adaptive))
    for a, b in zip(out[0][0], out[1][0]):
        for k in ("color", "depth", "hit_prim"):
            assert np.array_equal(getattr(a, k), getattr(b, k)), k
    _same(out[0][1], out[1][1])
