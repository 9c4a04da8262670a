"""A training step over several tiles per CTA and with the candidates in every
form that the tensor-core kernels take them: fewer and more per pixel than a
tile's stage holds (32), records that are 8- or only 4-byte aligned, cluster
counts that end within a thread's columns; against the FP64 oracle with the
kernels' BF16 roundings, as test_training_oracle.py (its tolerance)."""
import numpy as np
import pytest

import mlp_numpy
from test_training_oracle import TENSOR_KERNEL_TOLERANCE, blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,m,stride,phase,offset", [(256, 33, 1, 0, 1), (136, 40, 1, 0, 0), (16, 1, 1, 0, 1),
                                                     (248, 31, 2, 1, 0), (264, 35, 3, 2, 1)])
def test_gradient_matches_oracle(gpu, k, m, stride, phase, offset):
    import torch
    import risltc_gb300 as rl
    ctx = rl.Context(0)
    hs, offsets = rl.scenes.cluster_lights(
        rl.scenes.heightfield(230, 180, light_count=2400, triangle_count=0, seed=4, vertex_counts=(3, 8)), k, seed=3)
    n_lights, p = hs.light_count, hs.pixels
    light_cluster = np.repeat(np.arange(k), np.diff(offsets.astype(np.int64)))
    scene = rl.Scene.from_host_scene(ctx, hs)
    scene.set_clusters(offsets)
    model = rl.Model(ctx, k, seed=5)
    params = model.get_params()
    rng = np.random.default_rng(k)
    params[64 * 144 + 64 + 64 * 64 + 64:] *= 10.0
    model.set_params(params)
    center, half = (0.0, 0.0, 1.0), 6.0
    model.set_input_transform(center, half)
    scene.set_model(model)
    model.set_target_mix(0.5)
    lights = rng.integers(0, n_lights, (p, m)).astype(np.int32)
    weights = np.exp(rng.uniform(np.log(1e-3), np.log(10.0), (p, m))).astype(np.float32)
    weights[rng.uniform(size=(p, m)) < 0.1] = 0.0
    lights[rng.uniform(size=(p, m)) < 0.05] = n_lights
    flat = np.zeros(2 * p * m + offset, np.int32)
    flat[offset:] = np.stack([lights, weights.view(np.int32)], axis=2).ravel()
    d_cand = torch.from_numpy(flat).cuda()[offset:].view(p, m, 2)
    assert d_cand.data_ptr() % 8 == 4 * offset
    shaded = rng.uniform(0.0, 3.0, p).astype(np.float32)
    res = np.zeros((p, 4), np.int32)
    res[:, 0] = rng.integers(-1, n_lights, p)
    g = torch.from_numpy(hs.gbuffer).cuda()
    model.set_training_flags(accumulate_only=True)
    model.train(scene, g, hs.width, hs.height, d_cand, stride, phase, torch.from_numpy(shaded).cuda(),
                torch.from_numpy(res).cuda())
    got = model.get_gradient(clear=True)
    ctx.check()
    scene.close()
    model.close()
    ctx.close()
    train = np.arange(phase, p, stride)
    want = mlp_numpy.train_gradient(
        params, k, mlp_numpy.encode(hs.gbuffer[:, train], center, half), lights[train], weights[train], light_cluster,
        n_lights, np.float32(1.0) / np.float32(train.size), np.ones(train.size, bool), rounding="bf16",
        shaded=shaded[train], chosen=res[train, 0], shadowed_weight=0.5)
    for name, sl in blocks(k):
        scale = np.abs(want[sl]).max()
        assert scale > 0
        assert np.abs(got[sl] - want[sl]).max() <= TENSOR_KERNEL_TOLERANCE * scale, name
