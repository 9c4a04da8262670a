"""Model.logits into buffers of any alignment: whole 32-byte stores where the
caller's buffer allows them, single floats otherwise, the same bits either
way and nothing written outside; cluster counts below, at and past one
128-cluster product, pixel counts that leave a partial last tile."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters,pixels", [(8, 1), (72, 127), (128, 129), (136, 256), (1024, 131)])
def test_every_alignment_gives_the_same_logits(gpu, clusters, pixels):
    import torch
    import risltc_gb300 as rl
    from risltc_gb300 import _native
    ctx = rl.Context(0)
    model = rl.Model(ctx, clusters, seed=3)
    rng = np.random.default_rng(pixels)
    g = torch.from_numpy(rng.uniform(-1, 1, (17, pixels)).astype(np.float32)).cuda()
    want = model.logits(g, pixels, 1)
    assert want.data_ptr() % 32 == 0
    gb = _native.GBuffer(pixels, 1, g.data_ptr(), None)
    for offset in (1, 2, 4, 7):
        buf = torch.full((pixels * clusters + 16,), -7.5, device="cuda")
        at = buf.data_ptr() + 4 * offset
        _native.check(_native.load().risltc_model_logits(ctx.handle, model.handle, ctypes.byref(gb),
                                                         ctypes.c_void_p(at)), "risltc_model_logits")
        ctx.check()
        assert torch.equal(buf[offset:offset + pixels * clusters].view_as(want), want)
        assert (buf[:offset] == -7.5).all() and (buf[offset + pixels * clusters:] == -7.5).all()
    model.close()
    ctx.close()
