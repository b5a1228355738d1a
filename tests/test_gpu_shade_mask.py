"""The lighting step against the oracle: the masked light-probe sample for every probe
mask, with negative zeros, infinities and NaNs in the field, on the smallest and on odd
probe grids; the lights' reach for none, one, 31 and more lights, with frames of one
pixel, of part tiles and of whole ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(2, 2, 2), (3, 5, 2), (12, 12, 12)])
@pytest.mark.parametrize("special", [False, True])
def test_every_probe_mask(ctx, native, oracle_mod, res, special):
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=33, grid=24, n_spheres=6, n_lights=20, light_radius=5.0)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s)
    try:
        W, H = 133, 77
        pd = scenes.pass_data(s, W, H, lpf_res=res, aabb=(img.aabb[:3], img.aabb[3:]))
        cam, _, _ = ctx.trace_camera(sid, pd, native.CAM_PROB_MASK)
        rng = np.random.default_rng(sum(res))
        cam = cam.copy()
        cam[:, 5] = np.arange(len(cam)) % 256              # every mask
        field = rng.normal(0.0, 0.5, size=(7, res[2], res[1], res[0], 4)).astype(np.float16)
        if special:
            pick = rng.uniform(size=field.shape)
            field[pick < 0.10] = -0.0
            field[(pick > 0.10) & (pick < 0.15)] = 0.0
            field[(pick > 0.15) & (pick < 0.17)] = np.inf
            field[(pick > 0.17) & (pick < 0.19)] = -np.inf
            field[(pick > 0.19) & (pick < 0.20)] = np.nan
            field[(pick > 0.20) & (pick < 0.25)] = np.float16(6e-8)
        sh16 = field.view(np.uint16)
        out, f32, _ = ctx.shade_camera(sid, pd, cam, sh16, want_f32=True)
        o16, of32 = oracle_mod.shade_camera(oracle_mod.Scene(img, s.positions, s.normals), pd, cam, sh16)
        nan = np.isnan(of32)
        assert np.array_equal(np.isnan(f32), nan)
        assert np.array_equal(f32.view(np.uint32)[~nan], of32.view(np.uint32)[~nan])
        nan16 = np.isnan(o16.view(np.float16))
        assert np.array_equal(np.isnan(out.view(np.float16)), nan16)
        assert np.array_equal(out[~nan16], o16[~nan16])
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("size", [(1, 2), (31, 9), (33, 7), (64, 16), (257, 31)])
@pytest.mark.parametrize("n_lights,radius", [(0, 1.0), (1, 50.0), (31, 3.0), (40, 6.0)])
def test_lights_in_reach(ctx, native, oracle_mod, size, n_lights, radius):
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=34, grid=24, n_spheres=6, n_lights=n_lights, light_radius=radius)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s)
    try:
        pd = scenes.pass_data(s, *size, lpf_res=(4, 4, 4), aabb=(img.aabb[:3], img.aabb[3:]))
        cam, _, _ = ctx.trace_camera(sid, pd, 0)
        sh16 = np.random.default_rng(5).normal(0.0, 0.5, size=(7, 4, 4, 4, 4)).astype(np.float16).view(np.uint16)
        out, f32, _ = ctx.shade_camera(sid, pd, cam, sh16, want_f32=True)
        o16, of32 = oracle_mod.shade_camera(oracle_mod.Scene(img, s.positions, s.normals), pd, cam, sh16)
        assert np.array_equal(out, o16)
        assert np.array_equal(f32.view(np.uint32), of32.view(np.uint32))
    finally:
        ctx.free_scene(sid)
