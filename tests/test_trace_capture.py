"""risltc_trace_shadow captured into a CUDA graph and replayed on another stream
while the context traces on its own, around and past the ray count where
uncaptured calls share a cursor: every call answers every ray, replays with
other rays in the same buffer too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [-1, 1, 300001])
def test_replays_beside_the_contexts_own_calls(gpu, over):
    import torch
    import risltc_gb300 as rl
    count = torch.cuda.get_device_properties(0).multi_processor_count * 12 * 128 + over
    hs = rl.scenes.heightfield(32, 32, light_count=8, triangle_count=3000, seed=2)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    ctx = rl.Context(0, stream=stream.cuda_stream)
    scene = rl.Scene.from_host_scene(ctx, hs)

    def rays(seed):
        rng = np.random.default_rng(seed)
        r = np.zeros((count, 8), np.float32)
        r[:, 0:3] = rng.uniform((-6, -6, 0), (6, 6, 4), (count, 3))
        d = rng.normal(size=(count, 3))
        r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
        r[:, 3], r[:, 7] = 1e-3, rng.uniform(0.0, 12.0, count)
        return torch.from_numpy(r).cuda()

    a, b = rays(1), rays(2)
    want = []
    for r in (a, b):  # a few rays at a time: a thread per ray
        out = torch.full((count,), 7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for i in range(0, count, 100000):
            part, hit = r[i:i + 100000].contiguous(), out[i:i + 100000]
            torch.cuda.synchronize()
            rl.trace_shadow(ctx, scene, part, hit)
            ctx.check()
        want.append(out)
    buffer, replayed = a.clone(), torch.full((count,), 7, dtype=torch.int32, device="cuda")
    direct = torch.full((count,), 7, dtype=torch.int32, device="cuda")
    rl.trace_shadow(ctx, scene, a, direct)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        rl.trace_shadow(ctx, scene, buffer, replayed)
    for k in range(12):
        buffer.copy_((a, b)[k & 1])
        replayed.fill_(7)
        direct.fill_(7)
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            graph.replay()
        for _ in range(3):
            rl.trace_shadow(ctx, scene, b, direct)
        with torch.cuda.stream(other):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(replayed, want[k & 1]) and torch.equal(direct, want[1])
    ctx.check()
    scene.close()
    ctx.close()
