"""Uploads on either side of the sizes where another way makes the trees (the host, one
block, a launch a level), from images of any alignment, and what they leave allocated."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plain_bytes(img, s):
    leaf_tris = sum(int(img.leaf_words()[o]) & 0xFFF for o in img.nodes()[:, 3] if o != 0xFFFFFFFF)
    return img.data.nbytes + 2 * 12 * len(s.positions) + 16 * img.num_nodes + 48 * leaf_tris


def _check(native, oracle_mod, c, sid, img, s, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((6001, 8), np.float32)
    r[:, 0:3] = rng.uniform(0, 1, size=(6001, 3))
    d = rng.normal(size=(6001, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3] = 100.0
    r.view(np.uint32)[:, 7] = rng.integers(0, 2, 6001)
    sc = oracle_mod.Scene(img, s.positions, s.normals)
    for mode in (native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY):
        hit, nid, bary, _ = c.trace(sid, r, mode)
        oh, on, ob, _ = oracle_mod.trace(sc, r, mode)
        assert np.array_equal(hit, oh) and np.array_equal(nid, on)
        assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32))


# 2n - 1 nodes with one triangle a leaf: 3, 5, 767, 769, 8189 and 8193 of them
@pytest.mark.parametrize("tris,leaf", [(2, 1), (3, 1), (384, 1), (385, 1), (1100, 4), (4095, 1), (4097, 1), (1500, 15),
                                       (1000, 40)])
def test_trees_made_either_way(native, oracle_mod, tris, leaf):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(tris, tris)
    img = native.build_bvh(s, max_leaf_size=leaf)
    with native.Context(0) as c:
        for quant8 in (False, True):
            sid = c.upload(img, s, quant8=quant8)
            assert c.scene_bytes(sid) > _plain_bytes(img, s)   # the trees are there
            _check(native, oracle_mod, c, sid, img, s, tris)
            c.free_scene(sid)


@pytest.mark.parametrize("tris,leaf", [(300, 4), (2000, 1), (2000, 4), (30000, 1), (30000, 4)])
def test_an_upload_leaves_the_scene_alone_allocated(native, tris, leaf):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(1, tris)
    img = native.build_bvh(s, max_leaf_size=leaf)
    with native.Context(0) as c:
        before = c.memory_used()
        ids = [c.upload(img, s) for _ in range(3)]
        assert c.memory_used() == before + sum(c.scene_bytes(i) for i in ids)
        for i in ids:
            c.free_scene(i)
        assert c.memory_used() == before


@pytest.mark.parametrize("tris", [200, 3000])
def test_images_of_any_alignment(native, oracle_mod, tris):
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(7, tris)
    img = native.build_bvh(s)
    buf = np.zeros(img.data.nbytes + 64, np.uint8)
    off = (4 - buf.ctypes.data) % 16   # 4 bytes past a 16-byte boundary
    view = buf[off:off + img.data.nbytes]
    view[:] = np.frombuffer(img.data, np.uint8)
    odd = dataclasses.replace(img, data=view)
    with native.Context(0) as c:
        sid = c.upload(odd, s)
        _check(native, oracle_mod, c, sid, img, s, tris)


def test_bounds_of_the_vertices(native, oracle_mod):
    """The sort of a batch uses the scene's bounds: counts of vertices around a multiple of
    four, the least and the largest coordinate on any of them."""
    import torch
    from tim_raytracing_b200 import scenes
    with native.Context(0) as c:
        for tris in (1, 2, 3, 4, 5, 9):
            s = scenes.random_triangles(tris, tris)
            img = native.build_bvh(s)
            sid = c.upload(img, s)
            rng = np.random.default_rng(tris)
            r = np.zeros((500, 8), np.float32)
            r[:, 0:3] = rng.uniform(0, 1, size=(500, 3))
            r[:, 4:7] = s.positions[rng.integers(0, len(s.positions), 500)] - r[:, 0:3]
            r[:, 3] = 100.0
            want = oracle_mod.trace(oracle_mod.Scene(img, s.positions, s.normals), r, native.MODE_CLOSEST)[0]
            hit = torch.zeros((500, 4), dtype=torch.int32, device="cuda")
            c.set_launch_config(ray_sort=2)
            batch = c.batch_create([(sid, native.MODE_CLOSEST, 500, torch.from_numpy(r).cuda(), hit, None, None)])
            torch.cuda.synchronize()
            c.batch_launch(batch)
            torch.cuda.synchronize()
            assert np.array_equal(hit.cpu().numpy().view(np.uint32), want.view(np.uint32))
            c.batch_destroy(batch)


@pytest.mark.parametrize("tris", [3, 2000])
def test_triangles_out_of_reach(native, oracle_mod, tris):
    """The root's children are leaves without triangles; those of the image hang below them,
    where no walk goes. Both ways of making the trees have to see that there is nothing to
    make; one leaf with triangles beside an empty one makes them."""
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(tris, tris)
    img = native.build_bvh(s, max_leaf_size=1)
    words = img.leaf_words()
    zero = int(np.flatnonzero(words == 0)[0])   # a word that reads as a leaf of no triangles
    tri = next(int(o) for o in img.nodes()[:, 3] if o != 0xFFFFFFFF and int(words[o]) & 0xFFF)
    for offs in ((zero, zero), (tri, zero), (zero, tri)):
        data = np.array(img.data, copy=True)
        cut = dataclasses.replace(img, data=data)
        nodes = cut.nodes()
        left = int(nodes[0, 2]) & 0x3FFFFFFF
        nodes[0, 2] = left | 0xC0000000
        nodes[left:left + 2, 1] |= 0x80000000   # each other's sibling word says leaf too
        nodes[left, 3], nodes[left + 1, 3] = offs
        with native.Context(0) as c:
            sid = c.upload(cut, s)
            _check(native, oracle_mod, c, sid, cut, s, tris)
