"""Kernels whose work is split into tiles, at the edges of those: probe updates with
direction counts and probe ranges that are no multiple of what a block takes (64 rays, 8
probes), and GPU-built trees of sizes around a treelet's leaves and a block's warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_dirs", [1, 63, 65, 130])
@pytest.mark.parametrize("p0,p1", [(0, 1), (3, 12), (17, 64)])
def test_probe_sums(ctx, native, oracle_mod, num_dirs, p0, p1):
    from helpers import sh16_to_prev27
    from tim_raytracing_b200 import scenes
    O = oracle_mod
    s = scenes.heightfield_scene(seed=26, grid=24, n_spheres=5, n_lights=33, light_radius=4.0)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        res = (4, 4, 4)
        rng = np.random.default_rng(num_dirs)
        dirs = np.zeros((num_dirs, 4), np.float32)
        d = rng.normal(size=(num_dirs, 3))
        dirs[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
        basis = scenes.sh9_basis(dirs)
        lo, hi = img.aabb[:3], img.aabb[3:]
        sun, sunc = (-0.4, 0.3, -1.0), (1.0, 0.95, 0.9)
        prev16 = rng.uniform(-1, 1, size=(7, 4, 4, 4, 4)).astype(np.float16).view(np.uint16)
        sc, od = O.Scene(img, s.positions, s.normals), O.probe_desc(lo, hi, res, sun, sunc, num_dirs, 0.03)
        otr, oirr, _ = O.probe_trace(sc, od, dirs, p0, p1)
        osh = O.probe_sh9(od, basis, oirr.reshape(-1, 3), p0, p1, sh16_to_prev27(prev16, res, list(range(p0, p1))))
        for flags in (0, native.PROBE_WIDE):
            sh16 = prev16.copy()
            desc = native.probe_desc(lo, hi, res, sun, sunc, num_dirs, 0.03, flags)
            tr, irr, s32, _, _ = ctx.update_probes(sid, desc, dirs, basis, sh16, p0, p1, want_trace=True, want_irr=True,
                                                   want_sh32=True)
            assert np.array_equal(tr.reshape(-1), otr.reshape(-1))
            assert np.array_equal(irr.reshape(-1).view(np.uint32), oirr.reshape(-1).view(np.uint32))
            assert np.array_equal(s32.reshape(-1, 27).view(np.uint32), osh.view(np.uint32))
            assert np.array_equal(sh16_to_prev27(sh16, res, list(range(p0, p1))), osh.astype(np.float16).astype(np.float32))
            rest = [p for p in range(64) if not p0 <= p < p1]
            assert np.array_equal(sh16_to_prev27(sh16, res, rest), sh16_to_prev27(prev16, res, rest))
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("tris", [2, 3, 6, 7, 8, 9, 15, 33, 127, 128, 129, 1025])
@pytest.mark.parametrize("leaf", [1, 4])
def test_gpu_built_tree_sizes(ctx, native, oracle_mod, tris, leaf):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(40 + tris, tris)
    img = native.build_bvh(s, ctx=ctx, max_leaf_size=leaf)
    assert np.array_equal(img.data, native.build_bvh(s, ctx=ctx, max_leaf_size=leaf).data)
    rng = np.random.default_rng(tris)
    r = np.zeros((5000, 8), np.float32)
    r[:, 0:3] = rng.uniform(0, 1, size=(5000, 3))
    d = rng.normal(size=(5000, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3] = 100.0
    sid = ctx.upload(img, s, quant8=True)
    try:
        # the tree's own answers, and those of the host builder's tree: every triangle is in a
        # leaf (of two hits less than 1e-5 apart the one met first counts, so t may differ by that)
        oh, on, _, _ = oracle_mod.trace(oracle_mod.Scene(img, s.positions, s.normals), r, native.MODE_CLOSEST)
        host = native.build_bvh(s)
        hh, _, _, _ = oracle_mod.trace(oracle_mod.Scene(host, s.positions, s.normals), r, native.MODE_CLOSEST)
        t, th = oh[:, 3].copy().view(np.float32), hh[:, 3].copy().view(np.float32)
        assert np.array_equal(t < 100.0, th < 100.0) and np.abs(t - th).max() <= 1.1e-5
        for wide in (0, native.TRACE_WIDE):
            hit, nid, _, _ = ctx.trace(sid, r, native.MODE_CLOSEST | wide)
            assert np.array_equal(hit, oh) and np.array_equal(nid, on)
    finally:
        ctx.free_scene(sid)
