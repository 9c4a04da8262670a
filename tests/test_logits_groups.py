"""Model.logits over more tiles than the kernel has in flight: 128-pixel tiles
dealt to four, three, two or one group of warps per SM (the cluster count
decides how many fit), bulk and plain input loads, a partial last tile.  A
pixel's logits depend on its own inputs alone, so every pixel gets the bits of
a call on its tile alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters,pixels", [(256, 152 * 128 * 9 + 4), (256, 152 * 128 * 9 + 5), (512, 152 * 128 * 7 + 64),
                                             (640, 152 * 128 * 5 + 1), (1024, 152 * 128 * 2 + 100), (16, 152 * 128 + 8)])
def test_tiles_in_flight_do_not_mix(gpu, clusters, pixels):
    import torch
    import risltc_gb300 as rl
    ctx = rl.Context(0)
    model = rl.Model(ctx, clusters, seed=5)
    g = torch.from_numpy(np.random.default_rng(clusters).uniform(-1, 1, (17, pixels)).astype(np.float32)).cuda()
    got = model.logits(g, pixels, 1).view(pixels, clusters)
    ctx.check()
    tiles = (pixels + 127) // 128
    for tile in sorted({0, 1, 151, 152, 303, tiles // 2, tiles - 153, tiles - 2, tiles - 1}):
        if not 0 <= tile < tiles:
            continue
        part = g[:, 128 * tile:128 * (tile + 1)].contiguous()
        n = part.shape[1]
        assert torch.equal(got[128 * tile:128 * tile + n], model.logits(part, n, 1).view(n, clusters))
    # Every tile, against one call of a different tile-to-group assignment.
    half = (tiles // 2) * 128 // 4 * 4
    if half:
        a, b = g[:, :half].contiguous(), g[:, half:].contiguous()
        assert torch.equal(got[:half], model.logits(a, half, 1).view(half, clusters))
        assert torch.equal(got[half:], model.logits(b, pixels - half, 1).view(pixels - half, clusters))
    model.close()
    ctx.close()
