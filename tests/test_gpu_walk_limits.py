"""The walks of one kind of ray where little else tries them: rays without a range or an
origin in the binary form, against the oracle, and a frame with bounces (a pair of
overlapped launches) captured in a CUDA graph, against the frame itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rays_without_a_range_or_an_origin(ctx, native, oracle_mod):
    """tmax zero, negative, NaN and infinite; origins infinite, NaN and beyond every bound."""
    from tim_raytracing_b200 import scenes
    s = scenes.room_scene()
    img = native.build_bvh(s)
    leaf_tris = sum(int(img.leaf_words()[o]) & 0xFFF for o in img.nodes()[:, 3] if o != 0xFFFFFFFF)
    sid = ctx.upload(img, s)
    try:
        assert ctx.scene_bytes(sid) > img.data.nbytes + 24 * len(s.positions) + 16 * img.num_nodes + 48 * leaf_tris
        rng = np.random.default_rng(11)
        n = 40000
        r = np.zeros((n, 8), np.float32)
        r[:, 0:3] = rng.uniform((-1, -1, -1), (5, 5, 4), size=(n, 3))
        d = rng.normal(size=(n, 3))
        r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
        r[:, 4:7][rng.uniform(size=(n, 3)) < 0.1] = 0.0
        r[:, 3] = 100.0
        r.view(np.uint32)[:, 7] = rng.integers(0, 2, n)
        kind = rng.integers(0, 16, n)
        for k, t in enumerate((0.0, -0.0, -1.0, np.nan, np.inf, 1e-41)):
            r[kind == k, 3] = t
        axis = rng.integers(0, 3, n)
        for k, o in enumerate((np.inf, -np.inf, np.nan, 3e18, -2e12)):
            rows = np.flatnonzero(kind == 8 + k)
            r[rows, axis[rows]] = o
        sc = oracle_mod.Scene(img, s.positions, s.normals)
        for mode in (native.MODE_CLOSEST, native.MODE_ANY, native.MODE_PER_RAY):
            hit, nid, bary, _ = ctx.trace(sid, r, mode)
            oh, on, ob, _ = oracle_mod.trace(sc, r, mode)
            assert np.array_equal(hit.view(np.uint32), oh.view(np.uint32)), mode
            assert np.array_equal(nid, on), mode
            assert np.array_equal(bary.view(np.uint32), ob.view(np.uint32)), mode
    finally:
        ctx.free_scene(sid)


@pytest.mark.parametrize("wide", [False, True])
def test_a_captured_frame_with_bounces(ctx, native, wide):
    import torch
    from tim_raytracing_b200 import scenes
    s = scenes.heightfield_scene(seed=21, grid=24, n_spheres=4)
    img = native.build_bvh(s)
    sid = ctx.upload(img, s, quant8=True)
    try:
        w, h = 129, 67
        pd = scenes.pass_data(s, w, h, lpf_res=(8, 8, 8), aabb=(img.aabb[:3], img.aabb[3:]))
        flags = native.CAM_PROB_MASK | native.CAM_BOUNCE | (native.CAM_WIDE if wide else 0)
        out = torch.zeros((w * h, 8), dtype=torch.int32, device="cuda")
        bounce = torch.zeros((w * h, 4), dtype=torch.int32, device="cuda")
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        ctx.trace_camera_dev(sid, pd, flags, 5, None, None, out, bounce, stream=side.cuda_stream)
        torch.cuda.synchronize()
        want, want_bounce = out.cpu().numpy().copy(), bounce.cpu().numpy().copy()
        assert (want_bounce[:, 0:3] != 0).any()   # some bounces hit
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            ctx.trace_camera_dev(sid, pd, flags, 5, None, None, out, bounce, stream=side.cuda_stream)
        for _ in range(3):
            out.fill_(-1)
            bounce.fill_(-1)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)
            assert np.array_equal(bounce.cpu().numpy(), want_bounce)
        del graph
    finally:
        ctx.free_scene(sid)
