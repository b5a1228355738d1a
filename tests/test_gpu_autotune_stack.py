"""The autotuner leaves stack_depth as it is where the batch's launches don't read it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
def test_stack_depth_is_left_alone(native, wide):
    import torch
    from tim_raytracing_b200 import scenes
    s = scenes.random_triangles(4, 2000)
    img = native.build_bvh(s)
    rng = np.random.default_rng(1)
    rays = np.zeros((4000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(size=(4000, 3))
    rays[:, 3] = 10.0
    rays[:, 4:7] = rng.normal(size=(4000, 3))
    with native.Context(0) as c:
        sid = c.upload(img, s, quant8=True)
        d = torch.from_numpy(rays).cuda()
        hit = torch.zeros((4000, 4), dtype=torch.int32, device="cuda")
        batch = c.batch_create([(sid, native.MODE_ANY, 4000, d, hit, None, None)], wide=wide)
        torch.cuda.synchronize()
        for _ in range(8):
            c.set_launch_config(stack_depth=20)
            assert c.autotune_batch(batch, reps=1)["stack_depth"] == 20
            assert c.launch_config()["stack_depth"] == 20
        c.batch_destroy(batch)
