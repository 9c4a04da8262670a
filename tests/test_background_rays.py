"""Queues of 16 and more places per lane of a full grid, whose covered pixels are
numbered when the G-buffer has background (claims by shares), against calls that
number nothing: the candidate kernel of one thread per pixel notes no background.
Frames, running sums, reservoirs and ray counts bit for bit, with background in
rows above and below, scattered, everywhere but in one pixel, everywhere and
nowhere, one and three frames, sizes that leave partial warps; and the same in a
batch whose items mix these, also as a captured graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = ("none", "sky", "ground", "dots", "one", "all")


def primitives(pattern, w, h):
    p = np.zeros(w * h, np.uint32)
    if pattern == "sky":
        p[: w * (h * 2 // 3) + 5] = 0xFFFFFFFF
    elif pattern == "ground":
        p[w * (h // 3) + 7:] = 0xFFFFFFFF
    elif pattern == "dots":
        p[np.random.default_rng(w).uniform(size=w * h) < 0.7] = 0xFFFFFFFF
    elif pattern in ("one", "all"):
        p[:] = 0xFFFFFFFF
        if pattern == "one":
            p[w * h // 2] = 3
    return p


def large_enough(torch, places):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return places >= sms * 12 * 128 * 16


def buffers(torch, pixels):
    return (torch.full((pixels, 3), -1.0, device="cuda"), torch.full((pixels, 3), 0.5, dtype=torch.float64, device="cuda"),
            torch.full((pixels, 4), -7, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("w,h,frames", [(2049, 1001, 1), (1021, 641, 3)])
def test_frames_equal_those_without_numbers(gpu, w, h, frames):
    import torch
    import risltc_gb300 as rl
    assert large_enough(torch, 2 * w * h * frames)
    hs = rl.scenes.heightfield(w, h, light_count=60, triangle_count=2000, seed=3)
    ctx = rl.Context(0)
    scene = rl.Scene.from_host_scene(ctx, hs)
    g = torch.from_numpy(hs.gbuffer).cuda()
    for pattern in PATTERNS:
        prim = torch.from_numpy(primitives(pattern, w, h).view(np.int32)).cuda()
        got, want, rays = buffers(torch, w * h), buffers(torch, w * h), []
        for out, tile in ((want, "per_pixel"), (got, "32x8"), (got, "16x4")):
            out[1].fill_(0.5)
            rl.shade(ctx, scene, g, w, h, rl.settings(candidates=2, tile=tile), noise_seed=5, frames=frames,
                     out_rgb=out[0], accum=out[1], reservoirs=out[2], primitive=prim)
            ctx.check()
            rays.append(ctx.ray_count())
            if tile != "per_pixel":
                for a, b in zip(got, want):
                    assert torch.equal(a, b), (pattern, tile)
        assert rays[0] == rays[1] == rays[2] and (rays[0] == 0) == (pattern == "all")
    scene.close()
    ctx.close()


def test_batch_equals_single_calls(gpu):
    import torch
    import risltc_gb300 as rl
    stream = torch.cuda.Stream()
    ctx = rl.Context(0, stream=stream.cuda_stream)
    settings = rl.settings(candidates=2)
    items, want, places = [], [], 0
    with torch.cuda.stream(stream):
        for k, pattern in enumerate(PATTERNS):
            w, h, frames = 701 + 13 * k, 403 - 7 * k, 1 + k % 2
            hs = rl.scenes.heightfield(w, h, light_count=40, triangle_count=500 + 100 * k, seed=k)
            out, one = buffers(torch, w * h), buffers(torch, w * h)
            it = dict(scene=rl.Scene.from_host_scene(ctx, hs), gbuffer=torch.from_numpy(hs.gbuffer).cuda(), width=w,
                      height=h, settings=settings, noise_seed=9 + k, frames=frames, out_rgb=out[0], accum=out[1],
                      reservoirs=out[2], primitive=torch.from_numpy(primitives(pattern, w, h).view(np.int32)).cuda())
            rl.shade(ctx, it["scene"], it["gbuffer"], w, h, settings, noise_seed=9 + k, frames=frames, out_rgb=one[0],
                     accum=one[1], reservoirs=one[2], primitive=it["primitive"])
            items.append(it)
            want.append(one)
            places += 2 * w * h * frames
        extra = dict(items[0], **dict(zip(("out_rgb", "accum", "reservoirs"), buffers(torch, items[0]["width"] * items[0]["height"]))),
                     frames=3)  # takes the group past the border
        rl.shade_batch(ctx, items + [extra])
    assert large_enough(torch, places + 6 * items[0]["width"] * items[0]["height"])
    torch.cuda.synchronize()
    ctx.check()

    def check():
        for it, one in zip(items, want):
            assert torch.equal(it["out_rgb"], one[0]) and torch.equal(it["reservoirs"], one[2])
            assert torch.equal(it["accum"], one[1])
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        rl.shade_batch(ctx, items + [extra])
    for it in items:
        it["out_rgb"].fill_(-1.0)
        it["accum"].fill_(0.5)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    ctx.check()
    check()
    ctx.close()
