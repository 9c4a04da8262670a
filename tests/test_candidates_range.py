"""The candidate kernel's reservoirs at the ends of what its branch-free forms
cover, against the oracle bit for bit: scenes so small or so large that
squared lengths leave the square root's range (or are infinite), radiances
that take the candidates' weights out of the normal range, lights that fill
the hemisphere (edges of 90 degrees and more) or cross the horizon, every
vertex count, candidate counts that leave partial chunks and super-chunks, and
a light count that is no power of two."""
import numpy as np
import pytest

import golden_data as gd
from test_gpu_parity import gpu_render, oracle_render

pytestmark = pytest.mark.gpu

RIS = dict(technique="ltc_cp", light_sampling="ris", mis="optimal_clamped", sample_count=1, light_samples=1,
           fast_atan=False)


@pytest.fixture(scope="module")
def rl(gpu):
    import torch
    import risltc_gb300 as rl
    ctx = rl.Context(0)
    yield rl, ctx, torch
    ctx.close()


def scene(scale, radiance, lower, vertex_counts, count):
    """A heightfield frame with its lights lowered onto the surface, all
    lengths scaled and the radiance multiplied."""
    import risltc_gb300 as rlm
    hs = rlm.scenes.heightfield(61, 35, light_count=count, triangle_count=0, seed=13, vertex_counts=vertex_counts)
    g, lights = hs.gbuffer.copy(), hs.lights.copy()
    lights[:, 0:3] *= np.float32(radiance)
    for v in range(hs.max_vertex_count):
        lights[:, 14 + 4 * v] -= np.float32(lower)
    lights[:, 7] += lights[:, 6] * np.float32(lower)
    g[0:3] *= np.float32(scale)
    for v in range(hs.max_vertex_count):
        lights[:, 12 + 4 * v:15 + 4 * v] *= np.float32(scale)
    lights[:, 7] *= np.float32(scale)
    return dict(width=hs.width, height=hs.height, gbuffer=np.ascontiguousarray(g), primitive=hs.primitive,
                lights=lights, triangles=hs.triangles, max_vertex_count=hs.max_vertex_count)


@pytest.mark.parametrize("scale,radiance,lower,vertex_counts,count,candidates", [
    (1.0, 1.0, 3.0, (3, 8), 64, 33),       # lights in and below the surface: clips, wide edges
    (1.0, 1.0, 0.0, (3, 3), 100, 7),
    (1.0, 1.0, 2.5, (8, 8), 100, 9),
    (1e-13, 1.0, 1.0, (3, 8), 90, 32),     # squared lengths below 2^-76
    (1e-20, 1.0, 1.0, (3, 8), 64, 5),      # subnormal squared lengths
    (1e18, 1.0, 1.0, (3, 8), 90, 8),       # squared lengths near the largest number
    (1e20, 1.0, 1.0, (3, 8), 90, 8),       # infinite squared lengths
    (1.0, 1e-28, 1.0, (3, 8), 90, 40),     # weights below the normal test's range
    (1.0, 1e29, 1.0, (3, 8), 64, 40),      # weight sums above it, infinite p_hat
])
def test_reservoirs_equal_the_oracle(rl, scale, radiance, lower, vertex_counts, count, candidates):
    sc = scene(scale, radiance, lower, vertex_counts, count)
    c = dict(RIS, candidates=candidates)
    import risltc_gb300 as rlm
    with np.errstate(all="ignore"):
        _, _, idx, wp = gpu_render(rl, sc, c, noise_seed=5)
        _, ores, _ = oracle_render(sc, c, rlm.noise_constants(5)[0])
    assert np.array_equal(idx, ores["light_index"])
    assert np.array_equal(wp[:, 0], ores["w_sum"].astype(np.float32), equal_nan=True)
    assert np.array_equal(wp[:, 1], ores["sample_value"].astype(np.float32), equal_nan=True)
