"""The 8-wide form's walks of one kind of ray (any-hit, closest-hit) against the oracle,
where they can go wrong: batch sizes around a warp, leaves of one and of many triangles,
the smallest trees, coplanar duplicates (equal hits), components and origins on both sides
of what the box test is trusted for, tmax of every sort, and batches of several scenes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rays(rng, n, lo, hi, tmax=100.0):
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(lo, hi, size=(n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3] = tmax
    r.view(np.uint32)[:, 7] = rng.integers(0, 2, n)
    return r


def _check(native, oracle_mod, ctx, sid, sc, rays):
    for mode in (native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY):
        hit, nid, bary, _ = ctx.trace(sid, rays, mode | native.TRACE_WIDE)
        oh, on, ob, _ = oracle_mod.trace(sc, rays, mode)
        assert np.array_equal(hit.view(np.uint32), oh.view(np.uint32)), mode
        assert np.array_equal(nid, on), mode
        assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32)), mode
        hit, _, _, _ = ctx.trace(sid, rays, mode | native.TRACE_WIDE, want_nid=False, want_bary=False)
        assert np.array_equal(hit.view(np.uint32), oh.view(np.uint32)), mode


@pytest.mark.parametrize("n", [1, 31, 33, 1000, 65537])
def test_batch_sizes(ctx, native, oracle_mod, n):
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=21, grid=24, n_spheres=4)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        rng = np.random.default_rng(n)
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals),
               _rays(rng, n, (0, 0, 0), (20, 20, 6)))
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("n", [147, 1777, 5000, 14209, 37888, 37889])
def test_few_rays(ctx, native, oracle_mod, n):
    """Ray counts that are spread over the warps, one to eight to each, and just above, in
    both forms."""
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=23, grid=24, n_spheres=4)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        sc, rays = oracle_mod.Scene(img, s.positions, s.normals), _rays(np.random.default_rng(n), n, (0, 0, 0), (20, 20, 6))
        _check(native, oracle_mod, ctx, sid, sc, rays)
        for mode in (native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY):
            hit, nid, bary, _ = ctx.trace(sid, rays, mode)
            oh, on, ob, _ = oracle_mod.trace(sc, rays, mode)
            assert np.array_equal(hit.view(np.uint32), oh.view(np.uint32)), mode
            assert np.array_equal(nid, on), mode
            assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32)), mode
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("tris,leaf", [(1, 4), (2, 1), (3, 1), (9, 1), (40, 1), (3000, 15), (3000, 60)])
def test_leaf_sizes_and_small_trees(ctx, native, oracle_mod, tris, leaf):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(tris + leaf, tris)
    img = native.build_bvh(s, max_leaf_size=leaf)
    sid = ctx.upload(img, s, quant8=True)
    try:
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals),
               _rays(np.random.default_rng(leaf), 20000, 0.0, 1.0))
    finally:
        ctx.free_scene(sid)


def test_equal_hits(ctx, native, oracle_mod):
    """Each triangle several times over, as itself and moved by less than the offset that
    separates hits: the nearest hit is often not the binary walk's."""
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(4, 900)
    p = s.positions.reshape(-1, 3, 3)
    p[300:600] = p[:300]
    p[600:] = p[:300] + np.float32(3e-6)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals),
               _rays(np.random.default_rng(8), 40000, 0.0, 1.0))
    finally:
        ctx.free_scene(sid)


def test_directions_and_origins_on_the_margin(ctx, native, oracle_mod):
    """Zero, subnormal and tiny components (2^-57 to 2^-61 among them), long directions,
    origins on vertices' coordinates, far away and not finite, tmax from 1e-3 to infinity,
    zero, negative and NaN."""
    from tim_raytracing_b200 import scenes
    s = scenes.room_scene()
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        rng = np.random.default_rng(5)
        n = 60000
        r = _rays(rng, n, (-1, -1, -1), (5, 5, 4))
        z = rng.uniform(size=(n, 3))
        d = r[:, 4:7]
        d[z < 0.1] = 0.0
        d[(z > 0.1) & (z < 0.2)] *= np.float32(4e-8)
        tiny = (z > 0.2) & (z < 0.25)
        d[tiny] = np.ldexp(np.sign(d[tiny]), rng.integers(-61, -56, tiny.sum())).astype(np.float32)
        d[(z > 0.27) & (z < 0.28)] = np.float32(1e-41)
        d[rng.uniform(size=n) < 0.02] *= np.float32(1e12)
        on = rng.uniform(size=(n, 3)) < 0.3
        r[:, 0:3] = np.where(on, s.positions[rng.integers(0, len(s.positions), n)], r[:, 0:3])
        far = rng.uniform(size=n) < 0.05
        r[far, 0:3] *= np.float32(1e5)
        r[rng.uniform(size=n) < 0.002, 0] = np.float32(3e18)
        r[rng.uniform(size=n) < 0.002, 1] = np.float32(np.inf)
        r[:, 3] = np.where(rng.uniform(size=n) < 0.1, np.inf, np.exp(rng.uniform(-7, 12, n))).astype(np.float32)
        odd = rng.uniform(size=n)
        r[odd < 0.01, 3] = 0.0
        r[(odd > 0.01) & (odd < 0.02), 3] = -1.0
        r[(odd > 0.02) & (odd < 0.03), 3] = np.nan
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals), r)
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("modes", ["closest", "any", "mixed"])
@pytest.mark.parametrize("sort", [0, 1])
def test_batches_of_several_scenes(native, oracle_mod, modes, sort):
    """Both forms' batched walks, with scenes of which one has a single leaf (the 8-wide
    form then takes the general kernel) and without."""
    import torch
    from tim_raytracing_b200 import scenes
    with native.Context(0) as c:
        c.set_launch_config(ray_sort=sort)
        made = []
        for k, tris in enumerate((700, 50, 9, 2)):
            s = scenes.random_triangles(60 + k, tris)
            img = native.build_bvh(s, max_leaf_size=4)
            made.append((c.upload(img, s, quant8=True), oracle_mod.Scene(img, s.positions, s.normals)))
        rng = np.random.default_rng(17)
        M = {"closest": [native.MODE_CLOSEST], "any": [native.MODE_ANY],
             "mixed": [native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY]}[modes]
        for scenes_used in (made[:3], made):
            jobs, want = [], []
            for j in range(9):
                sid, sc = scenes_used[j % len(scenes_used)]
                rays, mode = _rays(rng, int(rng.integers(1, 3000)), 0.0, 1.0), M[j % len(M)]
                n = len(rays)
                jobs.append((sid, mode, n, torch.from_numpy(rays).cuda(), torch.zeros((n, 4), dtype=torch.int32, device="cuda"),
                             torch.zeros(n, dtype=torch.int32, device="cuda") if j % 2 else None,
                             torch.zeros((n, 2), dtype=torch.int32, device="cuda") if j % 2 else None))
                want.append(oracle_mod.trace(sc, rays, mode))
            for wide in (False, True):
                for job in jobs:
                    for out in job[4:]:
                        if out is not None:
                            out.fill_(7)
                batch = c.batch_create(jobs, wide=wide)
                torch.cuda.synchronize()
                c.batch_launch(batch)
                torch.cuda.synchronize()
                for (_, _, _, _, hit, nid, bary), (oh, on, ob, _) in zip(jobs, want):
                    assert np.array_equal(hit.cpu().numpy().view(np.uint32), oh.view(np.uint32))
                    if nid is not None:
                        assert np.array_equal(nid.cpu().numpy().view(np.uint32), on)
                        assert np.array_equal(bary.cpu().numpy().view(np.uint32), ob.view(np.uint32))
                c.batch_destroy(batch)
