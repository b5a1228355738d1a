"""Batches on 8-wide trees as deep as the walks of one kind of ray take (16 levels), and one
level deeper (the general kernel), against the oracle, with the deepest stacks that a launch
asks for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def deep_scene(seed):
    """400 triangles over eight decades of size around one point."""
    from tim_raytracing_b200 import scenes
    rng = np.random.default_rng(seed)
    k = 10.0 ** (-8.5 * rng.uniform(size=(400, 1, 1)))
    s = scenes.random_triangles(1, 400)
    s.positions[:] = (k * (rng.normal(size=(400, 1, 3)) + 0.05 * rng.normal(size=(400, 3, 3)))).reshape(-1, 3).astype(np.float32)
    return s


def deep_rays(rng, n):
    """Rays at points of every scale of the scene, from the same scales."""
    r = np.zeros((n, 8), np.float32)
    k = 10.0 ** (-8.5 * rng.uniform(size=(n, 2, 1)))
    o, to = (k * rng.normal(size=(n, 2, 3))).transpose(1, 0, 2)
    d = to - o
    r[:, 0:3] = o
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3] = 100.0
    r.view(np.uint32)[:, 7] = rng.integers(0, 2, n)
    return r


@pytest.mark.parametrize("seed,levels", [(29, 15), (4, 16), (0, 17)])
def test_batches_on_deep_trees(native, oracle_mod, seed, levels):
    import torch
    s = deep_scene(seed)
    img = native.build_bvh(s, max_leaf_size=1)
    assert native.wide_check(img, s.positions)["depth"] == levels
    sc = oracle_mod.Scene(img, s.positions, s.normals)
    with native.Context(0) as c:
        sid = c.upload(img, s, quant8=True)
        jobs, want = [], []
        for j, mode in enumerate((native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY)):
            rays = deep_rays(np.random.default_rng(10 + j), 3001)
            jobs.append((sid, mode, 3001, torch.from_numpy(rays).cuda(), torch.zeros((3001, 4), dtype=torch.int32, device="cuda"),
                         torch.zeros(3001, dtype=torch.int32, device="cuda"),
                         torch.zeros((3001, 2), dtype=torch.int32, device="cuda")))
            want.append(oracle_mod.trace(sc, rays, mode))
        assert any((w[1] != 0xFFFFFFFF).any() for w in want)   # some do hit
        for block in (64, 128, 256):
            c.set_launch_config(block=block)
            for wide in (False, True):
                batch = c.batch_create(jobs, wide=wide)
                torch.cuda.synchronize()
                c.batch_launch(batch)
                torch.cuda.synchronize()
                for (_, _, _, _, hit, nid, bary), (oh, on, ob, _) in zip(jobs, want):
                    assert np.array_equal(hit.cpu().numpy().view(np.uint32), oh.view(np.uint32))
                    assert np.array_equal(nid.cpu().numpy().view(np.uint32), on)
                    assert np.array_equal(bary.cpu().numpy().view(np.uint32), ob.view(np.uint32))
                c.batch_destroy(batch)
