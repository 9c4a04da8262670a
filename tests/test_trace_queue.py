"""risltc_trace_shadow around the ray count where it goes from a thread per ray
to the persistent queue (152 SMs x 12 blocks x 128 rays), with odd counts, rays
along the axes (infinite reciprocals), empty intervals and zero directions:
every ray's answer is that of a call on a few rays, which never queues, and of
the CPU's brute force over all triangles on a part of them."""
import ctypes

import numpy as np
import oracle
import pytest

pytestmark = pytest.mark.gpu

RESIDENT = 152 * 12 * 128


def scene_and_rays(count):
    rng = np.random.default_rng(17)
    import risltc_gb300 as rl
    hs = rl.scenes.heightfield(32, 32, light_count=8, triangle_count=3000, seed=2)
    rays = np.zeros((count, 8), np.float32)
    rays[:, 0:3] = rng.uniform((-6, -6, 0), (6, 6, 4), (count, 3))
    d = rng.normal(size=(count, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    axis = rng.uniform(size=count) < 0.2
    one = np.eye(3)[rng.integers(0, 3, count)] * rng.choice((-1.0, 1.0), count)[:, None]
    d[axis] = one[axis]
    two = rng.uniform(size=count) < 0.1
    d[two, rng.integers(0, 3, count)[two]] = 0.0
    d[rng.uniform(size=count) < 0.01] = 0.0
    rays[:, 4:7] = d
    rays[:, 3] = 1e-3
    rays[:, 7] = rng.uniform(0.0, 12.0, count)
    empty = rng.uniform(size=count) < 0.05
    rays[empty, 7] = rays[empty, 3]
    return hs, rays


@pytest.mark.parametrize("count", [RESIDENT - 1, RESIDENT, RESIDENT + 1, 2 * RESIDENT + 77])
def test_queue_answers_like_a_thread_per_ray(gpu, count):
    import torch
    import risltc_gb300 as rl
    hs, rays = scene_and_rays(count)
    ctx = rl.Context(0)
    scene = rl.Scene.from_host_scene(ctx, hs)
    d_rays = torch.from_numpy(rays).cuda()
    hits = torch.full((count,), 7, dtype=torch.int32, device="cuda")
    rl.trace_shadow(ctx, scene, d_rays, hits)
    want = torch.full((count,), 7, dtype=torch.int32, device="cuda")
    step = 100003
    for a in range(0, count, step):
        part = d_rays[a:a + step].contiguous()
        out = torch.full((part.shape[0],), 7, dtype=torch.int32, device="cuda")
        rl.trace_shadow(ctx, scene, part, out)
        want[a:a + step] = out
    ctx.check()
    scene.close()
    ctx.close()
    assert torch.equal(hits, want)
    some = np.flatnonzero((rays[:, 4:7] != 0).any(1))[::max(1, count // 20000)]
    lib = oracle.load()
    lib.oracle_f32_any_hit_omp.argtypes = [ctypes.POINTER(oracle.Scene), ctypes.c_void_p, ctypes.c_uint32,
                                           ctypes.c_void_p]
    osc = oracle.OracleScene(hs.lights, hs.max_vertex_count, hs.ltc0, hs.ltc1, hs.ltc_constants,
                             oracle.triangles_v0e1e2(hs.triangles))
    part = np.ascontiguousarray(rays[some])
    brute = np.zeros(some.size, np.uint32)
    lib.oracle_f32_any_hit_omp(ctypes.byref(osc.struct), part.ctypes.data, some.size, brute.ctypes.data)
    assert np.array_equal(hits.cpu().numpy()[some].astype(np.uint32), brute)
    assert ((hits == 0) | (hits == 1)).all() and 0.05 < hits.float().mean().item() < 0.95
