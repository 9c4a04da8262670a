"""The uniform-light estimator's scratch at its limits: a size that finds no
memory runs without it, keeps the smaller block and is not tried again; another
allocation that finds no memory takes the block's place and succeeds; results
stay those of a fresh context in every case.  The failing allocations are made
on the host (Context.inject_fault).  The same call in fast numerics, whose
estimator is the exact one, on both of its routes."""
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


def make(rl, torch, ctx, w, h):
    hs = rl.scenes.heightfield(w, h, light_count=30, triangle_count=300, seed=w)
    return dict(scene=rl.Scene.from_host_scene(ctx, hs), gbuffer=torch.from_numpy(hs.gbuffer).cuda(), width=w, height=h)


def shade(env, ctx, it, frames=1, **kw):
    rl, torch, stream, _ = env
    settings = rl.settings(**{**dict(light_sampling="uniform", candidates=1), **kw})
    with torch.cuda.stream(stream):
        out = torch.full((it["width"] * it["height"], 3), -1.0, device="cuda")
        rl.shade(ctx, it["scene"], it["gbuffer"], it["width"], it["height"], settings, noise_seed=4, frames=frames,
                 out_rgb=out)
    ctx.check()
    return out.cpu().numpy()


def test_a_size_without_memory_runs_without_the_queue(env):
    rl, torch, stream, ctx = env
    fresh = rl.Context(0, stream=stream.cuda_stream)
    small, large = make(rl, torch, ctx, 40, 30), make(rl, torch, ctx, 90, 70)
    want_small, want_large = (shade(env, fresh, make(rl, torch, fresh, *s)) for s in ((40, 30), (90, 70)))
    assert fresh.ray_count() > 0
    assert np.array_equal(shade(env, ctx, small), want_small)
    count = ctx.ray_count()
    assert count > 0
    ctx.inject_fault(allocation=True, allocation_retry=True)
    assert np.array_equal(shade(env, ctx, large), want_large)
    assert ctx.ray_count() == 0
    # Not tried again, though there is memory; the smaller block is back.
    assert np.array_equal(shade(env, ctx, large), want_large)
    assert ctx.ray_count() == 0
    ctx.inject_fault(allocation=True)  # for the next allocation, which no small call makes
    assert np.array_equal(shade(env, ctx, small), want_small)
    assert ctx.ray_count() == count
    fresh.close()


def test_growing_past_its_own_block(env):
    """No memory for the larger block beside the smaller: the smaller one goes first."""
    rl, torch, stream, ctx = env
    small, large = make(rl, torch, ctx, 40, 30), make(rl, torch, ctx, 90, 70)
    shade(env, ctx, small)
    ctx.inject_fault(allocation=True)
    got = shade(env, ctx, large)
    assert ctx.ray_count() > 0
    fresh = rl.Context(0, stream=stream.cuda_stream)
    assert np.array_equal(got, shade(env, fresh, make(rl, torch, fresh, 90, 70)))
    fresh.close()


def test_another_allocation_takes_the_blocks_memory(env):
    rl, torch, stream, ctx = env
    big = make(rl, torch, ctx, 1024, 512)
    want_uniform = shade(env, ctx, big, frames=2)
    count = ctx.ray_count()
    before = torch.cuda.mem_get_info()[0]
    # Scene creation allocates: the block goes, the scene comes.
    ctx.inject_fault(allocation=True)
    it = make(rl, torch, ctx, 40, 30)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] - before > 100 << 20  # 153 MB less the small scene's
    assert ctx.ray_count() == count  # still the last call's
    assert np.array_equal(shade(env, ctx, big, frames=2), want_uniform)
    assert ctx.ray_count() == 0  # that size was given up
    got = shade(env, ctx, it, light_sampling="ris", candidates=4)
    small = shade(env, ctx, it)
    assert ctx.ray_count() > 0  # a smaller one is not
    fresh = rl.Context(0, stream=stream.cuda_stream)
    other = make(rl, torch, fresh, 40, 30)
    assert np.array_equal(got, shade(env, fresh, other, light_sampling="ris", candidates=4))
    assert np.array_equal(small, shade(env, fresh, other))
    # Without a block to give up the failure is the caller's.
    fresh.close()
    bare = rl.Context(0, stream=stream.cuda_stream)
    bare.inject_fault(allocation=True)
    with pytest.raises(rl.RisltcError):
        make(rl, torch, bare, 40, 30)
    shade(env, bare, make(rl, torch, bare, 40, 30))
    bare.close()


@pytest.mark.parametrize("technique", ["ltc_cp", "projected_solid_angle"])
def test_fast_numerics_take_the_same_route(env, technique):
    rl, torch, stream, ctx = env
    it = make(rl, torch, ctx, 61, 35)
    want = shade(env, ctx, it, frames=2, technique=technique)
    got = shade(env, ctx, it, frames=2, technique=technique, numerics="fast")
    assert ctx.ray_count() > 0 and np.array_equal(got, want)
    out = torch.zeros((61 * 35, 3), device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        rl.shade(ctx, it["scene"], it["gbuffer"], 61, 35,
                 rl.settings(light_sampling="uniform", candidates=1, technique=technique, numerics="fast"), noise_seed=4,
                 frames=2, out_rgb=out)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
