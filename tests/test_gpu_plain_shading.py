"""The shading kernel without the principled, coarse-grid, AOV and edge code
against the oracle and against the full kernel, which a principled sphere out
of sight selects, at AO and shadow sample counts that start and end within a
word of the visibility flags."""
import numpy as np
import pytest

from parity import agree_mask_final, id_agreement, psnr_linear
from umbreon_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _render(ctx, sc, opt):
    b = ctx.build(sc)
    try:
        return ctx.render(b, sc, opt)
    finally:
        b.release()


@pytest.mark.parametrize("ao,shadow", [(0, 1), (0, 5), (1, 1), (2, 3), (3, 1), (5, 4), (7, 2), (16, 1), (33, 4)])
def test_plain_equals_full_and_oracle(gpu_ctx, oracle_lib, ao, shadow):
    sc, opt = scenes.ball_and_stick(n=700, width=96, height=54, supersample=2, ao_samples=ao)
    opt.shadows, opt.shadowSamples, opt.lightRadius = True, shadow, 3.0 if shadow > 1 else 0.0
    plain = _render(gpu_ctx, sc, opt)
    o = oracle_lib.render(sc, opt)
    # the grid parity tests' bars
    assert id_agreement(plain.hit_geom, plain.hit_prim, o.hit_geom, o.hit_prim) >= 0.999
    m = agree_mask_final(plain.hit_geom, plain.hit_prim, o.hit_geom, o.hit_prim, opt.supersample)
    assert np.quantile(np.abs(plain.color - o.color)[m], 0.999) <= 1e-3
    assert psnr_linear(plain.color, o.color) >= 45.0
    far = np.asarray(sc.camera.position) - 50.0 * np.asarray(sc.camera.direction)
    sc.sphere_center_radius = np.concatenate([sc.sphere_center_radius, [[*far, 1e-4]]]).astype(np.float32)
    sc.sphere_color = np.concatenate([sc.sphere_color, np.ones((1, 4))]).astype(np.float32)
    pbr = np.full(1, scenes.pov_material(), abi.MATERIAL_DTYPE)
    pbr["model"] = 1
    sc.sphere_material = np.concatenate([sc.sphere_material, pbr])
    full = _render(gpu_ctx, sc, opt)
    assert np.array_equal(plain.hit_prim, full.hit_prim)
    assert np.array_equal(plain.color, full.color)


def test_replayed_frames_follow_the_materials(gpu_ctx):
    """A material that only a parameter of the table changes: the frame's
    recorded launches are those of the new scene."""
    pics = []
    for model in (0, 1, 0, 1):
        sc, opt = scenes.ball_and_stick(n=300, width=64, height=48, supersample=1, ao_samples=4)
        sc.sphere_material = sc.sphere_material.copy()
        sc.sphere_material["model"] = model
        sc.sphere_material["pbr_metallic"] = 1.0
        sc.sphere_material["pbr_roughness"] = 0.3
        pics.append(_render(gpu_ctx, sc, opt).color.copy())
    assert not np.array_equal(pics[0], pics[1])
    assert np.array_equal(pics[0], pics[2]) and np.array_equal(pics[1], pics[3])
