"""A frame replayed from a captured graph is the frame its options ask for: one
built scene rendered again and again on one context, the denoiser's options (and
others that choose launches) changing in between, against a context that
launches every kernel on its own."""
import copy

import numpy as np
import pytest

from umbreon_gb300 import scenes
from umbreon_gb300.api import Context

pytestmark = pytest.mark.gpu

STEPS = [dict(), dict(denoiser=1), dict(), dict(denoiser=1), dict(denoiser=1, denoiseIters=1),
         dict(denoiser=2, denoiseIters=5), dict(denoiser=1, denoiseSigmaN=4.0), dict(denoiser=1, denoiseSigmaL=0.5),
         dict(denoiser=1, denoiseDemodulateAlbedo=False), dict(denoiser=1, denoiseIters=0), dict(aoWriteAov=False),
         dict(denoiser=1), dict(width=131, height=88, denoiser=1), dict(denoiser=1)]


def test_replayed_frames_follow_the_denoiser():
    sc, opt = scenes.molecular_surface(n_atoms=60, box=12.0, n_spheres=30, grid=1.0, width=67, height=41, ao_samples=4)
    sc.mesh_colors[:, 3] = 1.0  # opaque: one layer, the frames that are captured
    sc.assumedGamma = 1.8
    opt.aoWriteAov = True
    graphs, plain = Context(0), Context(0, graphs=False)
    a, b = graphs.build(sc), plain.build(sc)
    seen = set()
    for k, kw in enumerate(STEPS):
        o = copy.copy(opt)
        for name, v in kw.items():
            setattr(o, name, v)
        got, want = graphs.render(a, sc, o), plain.render(b, sc, o)
        assert got.stats["layers"] == 1
        assert np.array_equal(got.color, want.color), (k, kw)
        seen.add(want.color.tobytes())
    # the options do change the picture: none, the defaults, one iteration, either
    # sigma, no demodulation, the other size
    assert len(seen) == 7
    for x in (a, b):
        x.release()
    for x in (graphs, plain):
        x.close()
