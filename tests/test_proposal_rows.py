"""The learned proposal at cluster counts whose rows do not fill a warp's 32
blocks of 8 logits (232, 240, 248) and at their neighbours: a pixel's
candidates depend on its own logits alone.  Its reservoir and colour keep their
bits when the next pixels' inputs change so far that their logits exceed its
own by hundreds, and the last pixel's do when the same context shaded a larger
frame of such pixels before (the row past its own then holds stale logits).
Every second pixel's logits are spread over the clusters, so that a maximum
taken over a foreign row would leave all of its weights zero."""
import numpy as np
import pytest

import golden_data as gd

pytestmark = pytest.mark.gpu

FEATURES, HIDDEN = 144, 64
QUIET, LOUD = -0.75, 0.9375  # normalised x (exact in BF16): ReLU(x) gates the loud logits


def parameters(clusters):
    """Logits 2 sin(k) for a pixel with x < 0, 512 more in the first 24
    clusters for one with x > 0."""
    rng = np.random.default_rng(clusters)
    w1, w2 = np.zeros((HIDDEN, FEATURES), np.float32), np.zeros((HIDDEN, HIDDEN), np.float32)
    w3 = np.zeros((clusters, HIDDEN), np.float32)
    w1[0, 0] = 1.0
    w2[0, 0] = 1.0
    w3[:24, 0] = 512.0
    b3 = (2.0 * np.sin(np.arange(clusters)) + rng.uniform(-0.5, 0.5, clusters)).astype(np.float32)
    zero = np.zeros(HIDDEN, np.float32)
    return np.concatenate([w1.ravel(), zero, w2.ravel(), zero, w3.ravel(), b3])


@pytest.mark.parametrize("clusters", [224, 232, 240, 248, 256])
def test_candidates_depend_on_the_pixels_own_logits(gpu, clusters):
    import torch
    import risltc_gb300 as rl
    w, h = 37, 5
    pixels = w * h
    hs = rl.scenes.heightfield(w, h, light_count=2 * clusters, triangle_count=0, seed=4)
    l0, l1, k = gd.ltc()
    ctx = rl.Context(0)
    scene = rl.Scene(ctx, hs.lights, hs.max_vertex_count, l0, l1, k)
    scene.set_clusters(np.arange(0, 2 * clusters + 1, 2, dtype=np.uint32))
    model = rl.Model(ctx, clusters, seed=1)
    model.set_params(parameters(clusters))
    model.set_input_transform((0.0, 0.0, 0.0), 1.0)
    scene.set_model(model)
    settings = rl.settings(candidates=16, proposal="learned", proposal_uniform_fraction=0.05)

    def frame(height, loud):
        """The scene's G-buffer rows repeated to `height`, x as the network
        sees it QUIET, or LOUD where `loud`."""
        g = np.tile(hs.gbuffer.reshape(17, h, w), (1, (height + h - 1) // h, 1))[:, :height].reshape(17, -1).copy()
        g[0] = np.where(loud, LOUD, QUIET)
        return torch.from_numpy(np.ascontiguousarray(g)).cuda()

    def shade(g, height):
        out = torch.zeros((w * height, 3), device="cuda")
        res = torch.zeros((w * height, 4), dtype=torch.int32, device="cuda")
        rl.shade(ctx, scene, g, w, height, settings, noise_seed=3, out_rgb=out, reservoirs=res)
        ctx.check()
        return out.cpu().numpy().view(np.uint32), res.cpu().numpy()

    quiet = np.arange(pixels) % 2 == 0  # the last pixel too
    assert pixels % 2 == 1
    alone = frame(h, np.zeros(pixels, bool))
    mixed = frame(h, ~quiet)
    logits = model.logits(mixed, w, h).cpu().numpy().astype(np.float64)
    # The first 8, 16 and 24 logits of the following row (what a block past the
    # row would read) exceed the row's own by more than exp's range.
    own = logits.max(axis=1)[:-1][quiet[:-1]]
    assert (logits[1:, :24].min(axis=1)[quiet[:-1]] - own > 150.0).all()
    rgb0, res0 = shade(alone, h)
    rgb1, res1 = shade(mixed, h)
    assert np.array_equal(res0[quiet], res1[quiet]) and np.array_equal(rgb0[quiet], rgb1[quiet])
    assert not np.array_equal(res0[~quiet], res1[~quiet])
    # Stale loud logits behind the last pixel's row.
    shade(frame(2 * h, np.ones(2 * pixels, bool)), 2 * h)
    rgb2, res2 = shade(alone, h)
    assert np.array_equal(res0, res2) and np.array_equal(rgb0, rgb2)
    # The draws are the model's: not those of the uniform fallback.
    plain = rl.settings(candidates=16, proposal="learned", proposal_uniform_fraction=1.0)
    out = torch.zeros((pixels, 3), device="cuda")
    res = torch.zeros((pixels, 4), dtype=torch.int32, device="cuda")
    rl.shade(ctx, scene, alone, w, h, plain, noise_seed=3, out_rgb=out, reservoirs=res)
    assert not np.array_equal(res.cpu().numpy(), res0)
    scene.close()
    model.close()
    ctx.close()
