"""The reference's ground-truth estimator (one uniformly drawn light) with its
shadow rays queued, against the oracle bit for bit: every technique and MIS
heuristic that takes this route, background pixels, several frames, more
frames and then fewer (the scratch is larger than the call needs), a scene
with more lights than the one before, and a call captured into a CUDA graph
(which runs the fused kernel) against the direct call."""
import numpy as np
import pytest

import golden_data as gd
from test_gpu_parity import oracle_render

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(gpu):
    import torch
    import risltc_gb300 as rl
    stream = torch.cuda.Stream()
    ctx = rl.Context(0, stream=stream.cuda_stream)
    yield rl, torch, stream, ctx
    ctx.close()


def make(rl, torch, ctx, w, h, lights, seed):
    hs = rl.scenes.heightfield(w, h, light_count=lights, triangle_count=400, seed=seed, vertex_counts=(3, 8))
    hs.primitive[::7] = 0xFFFFFFFF
    sc = dict(width=w, height=h, gbuffer=hs.gbuffer, primitive=hs.primitive, lights=hs.lights, triangles=hs.triangles,
              max_vertex_count=hs.max_vertex_count)
    l0, l1, k = gd.ltc()
    scene = rl.Scene(ctx, hs.lights, hs.max_vertex_count, l0, l1, k, hs.triangles)
    g = torch.from_numpy(hs.gbuffer).cuda()
    prim = torch.from_numpy(hs.primitive.view(np.int32)).cuda()
    torch.cuda.synchronize()
    return sc, scene, g, prim


def render(env, made, s, frames=1, seed=3):
    rl, torch, stream, ctx = env
    sc, scene, g, prim = made
    p = sc["width"] * sc["height"]
    with torch.cuda.stream(stream):
        out = torch.full((p, 3), -1.0, device="cuda")
        acc = torch.zeros((p, 3), dtype=torch.float64, device="cuda")
        res = torch.full((p, 4), -7, dtype=torch.int32, device="cuda")
        rl.shade(ctx, scene, g, sc["width"], sc["height"], s, noise_seed=seed, frames=frames, out_rgb=out, accum=acc,
                 reservoirs=res, primitive=prim)
    ctx.check()
    return out.cpu().numpy(), acc.cpu().numpy(), res.cpu().numpy()


@pytest.mark.parametrize("technique,mis", [("ltc_cp", "optimal_clamped"), ("projected_solid_angle", "balance"),
                                           ("projected_solid_angle_biased", "weighted"), ("ltc_cp", "optimal"),
                                           ("projected_solid_angle", "power")])
def test_frames_equal_the_oracle(env, technique, mis):
    rl, torch, stream, ctx = env
    for w, h, lights in ((67, 31, 20), (33, 17, 300)):
        made = make(rl, torch, ctx, w, h, lights, seed=lights)
        s = rl.settings(technique=technique, light_sampling="uniform", mis=mis, candidates=1)
        c = dict(technique=technique, light_sampling="uniform", mis=mis, candidates=1, sample_count=1,
                 light_samples=1, fast_atan=False)
        sums = np.zeros((w * h, 3))
        for f in range(3):
            rgb, _, res = render(env, made, s, seed=3 + f)
            want, ores, _ = oracle_render(made[0], c, rl.noise_constants(3 + f)[0])
            assert np.array_equal(rgb, want)
            assert np.array_equal(res[:, 0], ores["light_index"]) and not res[:, 1:].any()
            assert 0 < ctx.ray_count() <= 2 * int((made[0]["primitive"] == 0).sum())
            sums += want.astype(np.float64)
        _, acc, _ = render(env, made, s, frames=3)
        assert np.array_equal(acc, sums)
        made[1].close()


def test_captured_call_equals_the_direct_call(env):
    rl, torch, stream, ctx = env
    made = make(rl, torch, ctx, 61, 35, 50, seed=8)
    sc, scene, g, prim = made
    s = rl.settings(light_sampling="uniform", candidates=1)
    want, _, _ = render(env, made, s, frames=2)
    out = torch.zeros((61 * 35, 3), device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        rl.shade(ctx, scene, g, 61, 35, s, noise_seed=3, frames=2, out_rgb=out, primitive=prim)
    # A larger call moves the scratch; the graph does not refer to it.
    big = make(rl, torch, ctx, 120, 64, 400, seed=9)
    render(env, big, s, frames=4)
    graph.replay()
    torch.cuda.synchronize()
    ctx.check()
    assert np.array_equal(out.cpu().numpy(), want)
    scene.close()
    big[1].close()
