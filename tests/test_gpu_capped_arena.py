"""A context with an arena cap that leaves room runs what one without a cap runs:
as many launches per GI frame, an adjoint of about the same time, the same
frames and gradients; and at the tightest caps that a call is accepted with, the
same results in many small chunks."""
import numpy as np
import pytest

from umbreon_gb300 import abi, scenes
from umbreon_gb300.abi import UbrError
from umbreon_gb300.api import Context

pytestmark = pytest.mark.gpu


def _gi(w, h, ss=1, integrator=1, n=300, **kw):
    sc, opt = scenes.ball_and_stick(n=n, width=w, height=h, supersample=ss, ao_samples=0)
    opt.gi, opt.giIntegrator = True, integrator
    for k, v in kw.items():
        setattr(opt, k, v)
    return sc, opt


def _once(cap, sc, call):
    """call(ctx, built) on a fresh context; None where the cap is refused."""
    ctx = Context(0, arena_bytes=cap)
    try:
        b = ctx.build(sc)
        try:
            return call(ctx, b)
        finally:
            b.release()
    except UbrError as e:
        assert e.status == abi.UBR_OUT_OF_MEMORY
        return None
    finally:
        ctx.close()


def _tightest(sc, call, hi=1 << 28):
    lo = 0
    assert _once(hi, sc, call) is not None
    while hi - lo > max(64, hi // 4096):
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _once(mid, sc, call) is not None else (mid, hi)
    return hi


@pytest.mark.parametrize("kw", [dict(w=640, h=480), dict(w=320, h=180, ss=2, integrator=2),
                                dict(w=300, h=200, integrator=2, pt2Adaptive=True, giBounces=2)])
def test_gi_frames_have_their_launches(kw):
    sc, opt = _gi(**kw)
    frames = [_once(cap, sc, lambda ctx, b: [ctx.render(b, sc, opt) for _ in range(2)]) for cap in (0, 1 << 33)]
    for a, c in zip(*frames):
        assert a.stats["kernels"] == c.stats["kernels"]
        assert np.array_equal(a.color, c.color)


def test_adjoint_takes_its_time():
    sc, opt = scenes.differentiable(n=2000, res=512)
    d = np.random.default_rng(2).normal(size=(512, 512, 4)).astype(np.float32)

    def call(ctx, b):
        return min(ctx.adjoint(b, sc, opt, d)["stats"]["adjoint_ms"] for _ in range(5))

    # (the smallest workspace makes some 750 chunks of this frame, twenty times
    # the time and more)
    assert _once(1 << 33, sc, call) < 3.0 * _once(0, sc, call)


@pytest.mark.parametrize("kw", [dict(w=9, h=7), dict(w=37, h=29, ss=2, integrator=2),
                                dict(w=33, h=21, integrator=2, giBounces=3, pt1Spp=33),
                                dict(w=37, h=29, integrator=2, pt1Spp=70, pt2Rounds=2),
                                dict(w=37, h=29, integrator=2, pt2Adaptive=True, pt2AdaptiveThresh=0.01),
                                dict(w=160, h=90, integrator=1, pt1Spp=300)])
def test_gi_frames_at_tight_caps(kw):
    sc, opt = _gi(**kw)

    def call(ctx, b):
        first = ctx.render(b, sc, opt)
        again = ctx.render(b, sc, opt)
        assert np.array_equal(first.color, again.color)
        return again.color

    want = _once(0, sc, call)
    cap = _tightest(sc, call)
    for room in (0, 1 << 10, 1 << 14, 1 << 17, 1 << 20):
        assert np.array_equal(_once(cap + room, sc, call), want), room


@pytest.mark.parametrize("kw", [dict(), dict(ao=0), dict(ao=33), dict(gamma=1.8, ss=2), dict(interior=True)])
@pytest.mark.parametrize("size", [(1, 1), (61, 43), (200, 90)])
def test_gradients_at_tight_caps(size, kw):
    sc, opt = scenes.differentiable(n=400, res=size[0], ao_samples=kw.get("ao", 8))
    opt.height = size[1]
    opt.supersample = kw.get("ss", 1)
    sc.assumedGamma = kw.get("gamma", 1.0)
    d = np.random.default_rng(2).normal(size=(size[1], size[0], 4)).astype(np.float32)

    def call(ctx, b):
        return ctx.adjoint(b, sc, opt, d, interior_only=kw.get("interior", False))

    want = _once(0, sc, call)
    cap = _tightest(sc, call)
    for room in (0, 1 << 10, 1 << 14, 1 << 17, 1 << 20):
        got = _once(cap + room, sc, call)
        assert got["stats"]["samples"] == want["stats"]["samples"]
        for k in want:
            if k == "stats":
                continue
            x, y = np.asarray(want[k], np.float64), np.asarray(got[k], np.float64)
            # float sums of the same terms in another order (a sphere collects a
            # few thousand terms)
            scale = max(np.abs(x).max(initial=0.0), 1e-30)
            assert np.abs(x - y).max(initial=0.0) <= 2e-4 * scale, (k, room)


def test_calls_take_turns_under_a_cap():
    """Frames, GI frames, adjoints and scene builds on one context whose cap holds
    the largest of them: none is refused because of what an earlier one kept."""
    sc, opt = scenes.differentiable(n=2000, res=256, ao_samples=8)
    gsc, gopt = _gi(256, 192, integrator=2)
    d = np.random.default_rng(2).normal(size=(256, 256, 4)).astype(np.float32)
    free = Context(0)
    b, g = free.build(sc), free.build(gsc)
    want = [free.render(b, sc, opt).color, free.render(g, gsc, gopt).color]
    grad = free.adjoint(b, sc, opt, d)["sphere_radius"]
    for x in (b, g):
        x.release()
    free.close()
    need = [_tightest(sc, lambda ctx, x: ctx.render(x, sc, opt)), _tightest(gsc, lambda ctx, x: ctx.render(x, gsc, gopt)),
            _tightest(sc, lambda ctx, x: ctx.adjoint(x, sc, opt, d))]
    scenes_bytes = 1 << 21  # both scenes stay, and are far below this
    # a plane kept from a 256 x 256 frame serves a 256 x 192 one: 4 / 3 of its need
    ctx = Context(0, arena_bytes=max(need) * 4 // 3 + scenes_bytes)
    b, g = ctx.build(sc), ctx.build(gsc)
    assert b.info()["device_bytes"] + g.info()["device_bytes"] < scenes_bytes
    for _ in range(2):
        assert np.array_equal(ctx.render(g, gsc, gopt).color, want[1])
        r = ctx.adjoint(b, sc, opt, d)["sphere_radius"]
        assert np.abs(r - grad).max() <= 2e-4 * np.abs(grad).max()
        assert np.array_equal(ctx.render(b, sc, opt).color, want[0])
        ctx.build(sc).release()
    for x in (b, g):
        x.release()
    ctx.close()
