"""risltc_shade_batch in several groups of 8 items beside each other: 8 and 9
items (one group, a second of one item), 17, and 70 (more groups than streams,
so that a stream runs two of them), in two calls without a wait in between and
as a captured graph; every item equals its own risltc_shade call bit for bit,
and calls before and after the batch on the context's stream keep their order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,candidates", [(8, 8), (9, 8), (17, 33), (70, 5)])
def test_groups_equal_single_calls(gpu, count, candidates):
    import torch
    import risltc_gb300 as rl
    rng = np.random.default_rng(count)
    stream = torch.cuda.Stream()
    ctx = rl.Context(0, stream=stream.cuda_stream)
    settings = rl.settings(candidates=candidates)
    items = []
    with torch.cuda.stream(stream):
        for k in range(count):
            hs = rl.scenes.plane_of_quads(int(rng.integers(1, 90)), int(rng.integers(1, 60)), int(rng.integers(1, 200)),
                                          seed=70 + k, triangles=int(rng.integers(1, 600)))
            primitive = np.zeros(hs.pixels, np.uint32)
            primitive[:: 3 + k % 5] = 0xFFFFFFFF
            items.append(dict(scene=rl.Scene.from_host_scene(ctx, hs), gbuffer=torch.from_numpy(hs.gbuffer).cuda(),
                              primitive=torch.from_numpy(primitive.view(np.int32)).cuda(), width=hs.width,
                              height=hs.height, settings=settings, frames=1 + k % 2,
                              out_rgb=torch.zeros((hs.pixels, 3), device="cuda"),
                              reservoirs=torch.zeros((hs.pixels, 4), dtype=torch.int32, device="cuda")))

        def single(k, seed):
            it = items[k]
            rgb, res = torch.zeros_like(it["out_rgb"]), torch.zeros_like(it["reservoirs"])
            rl.shade(ctx, it["scene"], it["gbuffer"], it["width"], it["height"], settings, noise_seed=seed,
                     frames=it["frames"], out_rgb=rgb, reservoirs=res, primitive=it["primitive"])
            return rgb, res

        first = [single(k, 5 * k) for k in range(count)]
        second = [single(k, 5 * k + 1000) for k in range(count)]

        def batch(offset):
            return rl.shade_batch(ctx, [dict(it, noise_seed=5 * k + offset) for k, it in enumerate(items)])

        def equal(want):
            return all(torch.equal(it["out_rgb"], w[0]) and torch.equal(it["reservoirs"], w[1])
                       for it, w in zip(items, want))

        before = ctx.launch_count()
        batch(0)
        assert ctx.launch_count() - before == 4 * ((count + 7) // 8)
        kept = [it["out_rgb"].clone() for it in items]  # behind the batch on its stream
        batch(1000)
        after = single(0, 1000)
    torch.cuda.synchronize()
    ctx.check()
    assert all(torch.equal(a, w[0]) for a, w in zip(kept, first))
    assert equal(second) and torch.equal(after[0], second[0][0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        batch(0)
    for _ in range(2):
        for it in items:
            it["out_rgb"].fill_(-1.0)
            it["reservoirs"].fill_(-9)
        graph.replay()
        torch.cuda.synchronize()
        ctx.check()
        assert equal(first)
    ctx.close()
