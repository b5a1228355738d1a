"""Any-hit rays of the binary form whose walks leave more slots waiting than their stack
holds one by one (csrc/four_stack.h), in single and batched launches, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def needle_scene(n, length):
    """Long crossing needles: nearly every box on a ray's way is entered."""
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(3, n)
    rng = np.random.default_rng(6)
    p = rng.uniform(0, 1, size=(n, 1, 3)) + np.zeros((n, 3, 3))
    p[:, 1] += length * rng.normal(size=(n, 3))
    p[:, 2] = p[:, 1] + rng.normal(scale=1e-4, size=(n, 3))
    s.positions[:] = p.reshape(-1, 3).astype(np.float32)
    return s


def needle_rays(rng, n):
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(0, 1, size=(n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3] = 100.0
    r.view(np.uint32)[:, 7] = rng.integers(0, 2, n)
    return r


@pytest.mark.parametrize("n,length,leaf", [(20000, 1.0, 4), (3000, 1.0, 1), (60000, 0.1, 2)])
def test_walks_of_many_waiting_slots(native, oracle_mod, n, length, leaf):
    import torch
    s = needle_scene(n, length)
    img = native.build_bvh(s, max_leaf_size=leaf)
    sc = oracle_mod.Scene(img, s.positions, s.normals)
    rays = needle_rays(np.random.default_rng(n), 3001)
    want = {m: oracle_mod.trace(sc, rays, m) for m in (native.MODE_ANY, native.MODE_PER_RAY)}
    assert want[native.MODE_ANY][0][:, 0].any() and not want[native.MODE_ANY][0][:, 0].all()   # both answers occur
    with native.Context(0) as c:
        sid = c.upload(img, s)
        leaf_tris = sum(int(img.leaf_words()[o]) & 0xFFF for o in img.nodes()[:, 3] if o != 0xFFFFFFFF)
        plain = img.data.nbytes + 2 * 12 * len(s.positions) + 16 * img.num_nodes + 48 * leaf_tris
        assert c.scene_bytes(sid) > plain   # the trees are there
        for block in (64, 128, 256):
            c.set_launch_config(block=block)
            for mode, (oh, on, ob, _) in want.items():
                hit, nid, bary, _ = c.trace(sid, rays, mode)
                assert np.array_equal(hit, oh) and np.array_equal(nid, on)
                assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32))
            out = [(torch.zeros((3001, 4), dtype=torch.int32, device="cuda"), m) for m in want]
            d = torch.from_numpy(rays).cuda()
            batch = c.batch_create([(sid, m, 3001, d, h, None, None) for h, m in out])
            torch.cuda.synchronize()
            c.batch_launch(batch)
            torch.cuda.synchronize()
            for h, m in out:
                assert np.array_equal(h.cpu().numpy().view(np.uint32), want[m][0].view(np.uint32))
            c.batch_destroy(batch)
