"""risltc_ctx_ray_count and captured calls beside batches: the count is that of
the last risltc_shade call whatever batches ran since (fused ones, whose first
item traces another number of rays, and mixed ones, whose first item queues
none), and a captured call keeps its counters when a batch of more items than
any before comes between its capture and its replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def env(gpu):
    import torch
    import risltc_gb300 as rl
    stream = torch.cuda.Stream()
    ctx = rl.Context(0, stream=stream.cuda_stream)
    yield rl, torch, stream, ctx
    ctx.close()


def make(rl, torch, ctx, w, h, seed, triangles):
    hs = rl.scenes.plane_of_quads(w, h, 40, seed=seed, triangles=triangles)
    return dict(scene=rl.Scene.from_host_scene(ctx, hs), gbuffer=torch.from_numpy(hs.gbuffer).cuda(), width=w, height=h,
                out_rgb=torch.zeros((w * h, 3), device="cuda"), noise_seed=seed, frames=1)


def shade(rl, ctx, it, settings, out=None):
    rl.shade(ctx, it["scene"], it["gbuffer"], it["width"], it["height"], settings, noise_seed=it["noise_seed"],
             out_rgb=it["out_rgb"] if out is None else out)


def test_count_is_the_last_single_calls(env):
    rl, torch, stream, ctx = env
    default = rl.settings(candidates=4)
    other = rl.settings(technique="projected_solid_angle", candidates=4)
    with torch.cuda.stream(stream):
        one = make(rl, torch, ctx, 64, 48, 1, 400)
        small = [dict(make(rl, torch, ctx, 16 + k, 16, 2 + k, 300), settings=default) for k in range(11)]
    assert ctx.ray_count() == 0
    rl.shade_batch(ctx, small[:2])
    assert ctx.ray_count() == 0
    shade(rl, ctx, one, default)
    count = ctx.ray_count()
    assert 2 * 16 * 16 < count <= 2 * 64 * 48
    rl.shade_batch(ctx, small)  # more items than before, one launch per phase
    assert ctx.ray_count() == count
    mixed = [dict(small[0], settings=other)] + small + small
    rl.shade_batch(ctx, mixed)  # more items again, the first without a ray queue
    assert ctx.ray_count() == count
    ctx.check()
    shade(rl, ctx, one, rl.settings(candidates=4, shadows=False))
    assert ctx.ray_count() == 0


@pytest.mark.parametrize("triangles", [0, 400])
def test_a_captured_call_outlives_a_larger_batch(env, triangles):
    """The first batch sizes records, rays and p_hat slots; the second has
    fewer pixels and more items."""
    rl, torch, stream, ctx = env
    default = rl.settings(candidates=4)
    with torch.cuda.stream(stream):
        one = make(rl, torch, ctx, 96, 64, 1, triangles)
        big = [dict(make(rl, torch, ctx, 128, 96, 50 + k, 300), settings=default) for k in range(2)]
        small = [dict(make(rl, torch, ctx, 17, 16, 2 + k, 300), settings=default) for k in range(40)]
        out = torch.zeros((96 * 64, 3), device="cuda")
    rl.shade_batch(ctx, big)
    shade(rl, ctx, one, default)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        shade(rl, ctx, one, default, out)
    rl.shade_batch(ctx, small)
    torch.cuda.synchronize()  # the graph and the context share scratch: one after the other
    graph.replay()
    torch.cuda.synchronize()
    ctx.check()
    assert torch.equal(out, one["out_rgb"]) and (out != 0).any()
