"""The binary form's two walks (4-wide tree for any-hit rays, child-pair records for
closest-hit rays) against the oracle, where they can go wrong: batch sizes around a
warp, leaves of more than 15 triangles, the smallest trees, rays with zero or tiny
components and far origins, origins on box planes, walks that outgrow the any-hit
stack, and a context with a memory budget (which keeps the plain walk)."""
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
        hit, nid, bary, _ = ctx.trace(sid, rays, mode)
        oh, on, ob, _ = oracle_mod.trace(sc, rays, mode)
        assert np.array_equal(hit, oh), mode
        assert np.array_equal(nid, on), mode
        assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32)), mode
        hit, _, _, _ = ctx.trace(sid, rays, mode, want_nid=False, want_bary=False)
        assert np.array_equal(hit, oh), mode


@pytest.mark.parametrize("n", [1, 31, 33, 1000, 65537])
def test_batch_sizes(ctx, native, oracle_mod, n):
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=21, grid=24, n_spheres=4)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s)
    try:
        rng = np.random.default_rng(n)
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals),
               _rays(rng, n, (0, 0, 0), (20, 20, 6)))
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("tris,leaf", [(2, 1), (3, 1), (40, 1), (3000, 15), (3000, 16), (3000, 60)])
def test_leaf_sizes_and_small_trees(ctx, native, oracle_mod, tris, leaf):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(tris + leaf, tris)
    img = native.build_bvh(s, max_leaf_size=leaf)
    sid = ctx.upload(img, s)
    try:
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals),
               _rays(np.random.default_rng(leaf), 20000, 0.0, 1.0))
    finally:
        ctx.free_scene(sid)


def test_directions_and_origins_on_the_margin(ctx, native, oracle_mod):
    """Zero, subnormal and tiny components, origins on vertices' coordinates (box planes)
    and far away, tmax from 1e-3 to infinity."""
    from tim_raytracing_b200 import scenes
    s = scenes.room_scene()
    img = native.build_bvh(s)
    sid = ctx.upload(img, s)
    try:
        rng = np.random.default_rng(5)
        n = 60000
        r = _rays(rng, n, (-1, -1, -1), (5, 5, 4))
        z = rng.uniform(size=(n, 3))
        d = r[:, 4:7]
        d[z < 0.2] = 0.0
        d[(z > 0.2) & (z < 0.25)] *= np.float32(4e-8)
        d[(z > 0.25) & (z < 0.27)] *= np.float32(1e-20)
        d[(z > 0.27) & (z < 0.28)] = np.float32(1e-41)
        on = rng.uniform(size=(n, 3)) < 0.3
        r[:, 0:3] = np.where(on, s.positions[rng.integers(0, len(s.positions), n)], r[:, 0:3])
        far = rng.uniform(size=n) < 0.05
        r[far, 0:3] *= np.float32(1e5)
        r[rng.uniform(size=n) < 0.002, 0] = np.float32(3e12)   # beyond the any-hit test's range
        r[:, 3] = np.where(rng.uniform(size=n) < 0.1, np.inf, np.exp(rng.uniform(-7, 12, n))).astype(np.float32)
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals), r)
    finally:
        ctx.free_scene(sid)


def test_any_hit_walk_that_outgrows_its_stack(ctx, native, oracle_mod):
    """Long crossing needles: nearly every box is entered, so more slots wait than the
    any-hit stack holds and the plain walk answers."""
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(3, 20000)
    rng = np.random.default_rng(6)
    p = rng.uniform(0, 1, size=(20000, 1, 3)) + np.zeros((20000, 3, 3))
    p[:, 1] += rng.normal(size=(20000, 3))
    p[:, 2] = p[:, 1] + rng.normal(scale=1e-4, size=(20000, 3))
    s.positions[:] = p.reshape(-1, 3).astype(np.float32)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s)
    try:
        _check(native, oracle_mod, ctx, sid, oracle_mod.Scene(img, s.positions, s.normals), _rays(rng, 4000, 0.0, 1.0))
    finally:
        ctx.free_scene(sid)


def test_memory_budget_keeps_the_scene_size(native, oracle_mod):
    """With a memory budget a scene takes what it always took, and traces the same."""
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=22, grid=24, n_spheres=4)
    img = native.build_bvh(s)
    rays = _rays(np.random.default_rng(9), 20000, (0, 0, 0), (20, 20, 6))
    size = {}
    for budget in (0, 1 << 30):
        with native.Context(0, mem_budget_bytes=budget) as c:
            sid = c.upload(img, s)
            size[budget] = c.scene_bytes(sid)
            _check(native, oracle_mod, c, sid, oracle_mod.Scene(img, s.positions, s.normals), rays)
    leaf_tris = sum(int(img.leaf_words()[o]) & 0xFFF for o in img.nodes()[:, 3] if o != 0xFFFFFFFF)
    plain = img.data.nbytes + 2 * 12 * len(s.positions) + 16 * img.num_nodes + 48 * leaf_tris
    assert size[1 << 30] == plain
    assert size[0] > plain
