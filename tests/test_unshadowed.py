"""Default calls without shadow rays (one estimator kernel) against the same
calls with an occluder that no ray can reach (sample, trace and resolve
kernels): frames, running sums and reservoirs bit for bit, for every MIS
heuristic, background pixels, several frames, sizes below and past a warp, a
block and a warp per 32 pixels of the largest grid."""
import numpy as np
import pytest

import golden_data as gd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,frames,mis", [(1, 1, 2, "optimal_clamped"), (31, 1, 1, "balance"), (33, 3, 3, "power"),
                                            (129, 65, 1, "weighted"), (480, 270, 2, "optimal"),
                                            (701, 503, 2, "optimal_clamped")])
def test_estimator_kernel_equals_the_queued_one(gpu, w, h, frames, mis):
    import torch
    import risltc_gb300 as rl
    hs = rl.scenes.heightfield(w, h, light_count=50, triangle_count=0, seed=w, vertex_counts=(3, 8))
    primitive = np.zeros(w * h, np.uint32)
    primitive[5::7] = 0xFFFFFFFF
    far = np.array([[0, 0, -900, 1, 0, -900, 0, 1, -900]], np.float32)
    l0, l1, k = gd.ltc()
    ctx = rl.Context(0)
    g = torch.from_numpy(hs.gbuffer).cuda()
    prim = torch.from_numpy(primitive.view(np.int32)).cuda()

    def render(triangles, shadows):
        scene = rl.Scene(ctx, hs.lights, hs.max_vertex_count, l0, l1, k, triangles)
        out = torch.full((w * h, 3), -1.0, device="cuda")
        acc = torch.full((w * h, 3), 0.5, dtype=torch.float64, device="cuda")
        res = torch.full((w * h, 4), -7, dtype=torch.int32, device="cuda")
        before = ctx.launch_count()
        rl.shade(ctx, scene, g, w, h, rl.settings(candidates=5, mis=mis, shadows=shadows), noise_seed=11, frames=frames,
                 out_rgb=out, accum=acc, reservoirs=res, primitive=prim)
        ctx.check()
        launches = ctx.launch_count() - before
        scene.close()
        return out, acc, res, launches

    want = render(far, True)
    assert want[3] == 4
    for triangles, shadows in ((far, False), (np.zeros((0, 9), np.float32), True)):
        got = render(triangles, shadows)
        assert got[3] == 2
        for a, b in zip(got[:3], want[:3]):
            assert torch.equal(a, b)
    assert w * h == 1 or (want[0] != 0).any()
    ctx.close()
