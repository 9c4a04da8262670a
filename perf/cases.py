"""The work whose speed is followed: calls that users of this framework make.

A case is a dict of plain values.  Its "kind" names the entry point:

  frame   risltc_gb300.shade on device buffers: candidates, projected solid
          angle samples, shadow rays, resolve (and the proposal where the case
          has one)
  host    risltc_gb300.shade_host: the same from and to host memory
  batch   risltc_gb300.shade_batch: several scenes in one call
  logits  Model.logits: the learned proposal's forward pass for a frame
  train   Model.train and get_gradient: one training step's gradient
  rays    risltc_gb300.trace_shadow: any-hit queries of the caller's own

listed() holds the cases, draw() gives more of the same ranges, prepare() makes
what the caller has in hand, run() is one pass, work() what a pass cannot do
without and exact() the outputs in 64 bits where they have such a value.
"""
import functools
import math

import numpy as np
import torch

import risltc_gb300 as rl

# Operations per candidate and light vertex (both spaces), per pixel-frame's
# estimator and per pixel-frame's shadow rays: counts of the algorithm's
# floating-point operations on heightfield frames.
FLOPS_VERTEX, FLOPS_ESTIMATOR, FLOPS_RAYS = 130.0, 3000.0, 1700.0
FEATURES, HIDDEN = 144, 64
CENTER, HALF_EXTENT = (0.0, 0.0, 1.0), 6.0


def listed():
    return [
        # A tool's thumbnail through host buffers: the smallest call, where
        # launches, copies and waits count.
        dict(name="thumbnail_64_host", kind="host", scene="plane", width=64, height=64, lights=64, triangles=500,
             candidates=8, frames=1),
        # The smallest configuration of the benchmark: a plane lit by 64
        # quads, no occluders.
        dict(name="plane_256", kind="frame", scene="plane", width=256, height=256, lights=64, triangles=0,
             candidates=8, frames=1),
        # An interactive viewport: odd sizes, a candidate count and a light
        # count that are no power of two, another MIS heuristic, three frames.
        dict(name="viewport_961x541", kind="frame", scene="heightfield", width=961, height=541, lights=1000,
             triangles=3001, candidates=17, frames=3, mis="weighted"),
        # One frame of an animation at the reference's 32 candidates.
        dict(name="frame_1080p", kind="frame", scene="heightfield", width=1920, height=1080, lights=1024,
             triangles=200000, candidates=32, frames=1),
        # The many-lights frame of the benchmark's headline: four samples per
        # pixel in one call.
        dict(name="many_lights_1080p", kind="frame", scene="heightfield", width=1920, height=1080, lights=16384,
             triangles=1000000, candidates=32, frames=4),
        # The same kind of frame in fast numerics.
        dict(name="fast_720p", kind="frame", scene="heightfield", width=1280, height=720, lights=4096,
             triangles=100000, candidates=32, frames=2, numerics="fast"),
        # The learned proposal in use: a trained model steers 8 candidates.
        dict(name="learned_1080p", kind="frame", scene="heightfield", width=1920, height=1080, lights=16384,
             triangles=20000, candidates=8, frames=4, proposal="learned", clusters=256),
        # The reference's ground-truth estimator: one light drawn uniformly,
        # projected solid angle sampling, shadow rays.
        dict(name="uniform_640x360", kind="frame", scene="heightfield", width=640, height=360, lights=1024,
             triangles=5000, candidates=1, frames=4, light_sampling="uniform"),
        # Several small to large scenes of a render queue in one call.
        dict(name="batch_6_scenes", kind="batch", scene="plane", items=6, min_side=256, max_side=1400, lights=4096,
             triangles=200000, candidates=8, frames=1),
        # The proposal's forward pass for a 960x540 frame.
        dict(name="logits_960x540", kind="logits", scene="heightfield", width=960, height=540, clusters=256),
        # One online training step on every 16th pixel of a 1080p frame.
        dict(name="train_1080p", kind="train", scene="heightfield", width=1920, height=1080, lights=16384,
             clusters=256, candidates=32, stride=16),
        # A caller's own visibility queries.
        dict(name="rays_2m", kind="rays", lights=1024, triangles=200000, rays=2000000),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo, hi):  # a frame of about lo..hi pixels, 1:1 to 21:9
        n, aspect = log_int(lo, hi), rng.uniform(1.0, 2.33)
        h = max(8, int(math.sqrt(n / aspect)))
        return dict(width=max(8, n // h), height=h)

    kind = rng.choice(["host", "frame", "frame", "frame", "fast", "learned", "uniform", "batch", "logits", "train",
                       "rays"])
    if kind == "host":
        return dict(kind="host", scene="plane", **size(2000, 60000), lights=log_int(16, 1024),
                    triangles=log_int(100, 20000), candidates=rng.randint(1, 16), frames=1)
    if kind in ("frame", "fast"):
        scene = rng.choice(["plane", "heightfield", "heightfield"])
        case = dict(kind="frame", scene=scene, **size(30000, 2000000), lights=log_int(16, 16384),
                    triangles=rng.choice([0, 1, 1, 1]) * log_int(500, 300000), candidates=rng.randint(2, 32),
                    frames=rng.randint(1, 4))
        if kind == "fast":
            case["numerics"] = "fast"
        else:
            case["mis"] = rng.choice(["optimal_clamped", "optimal_clamped", "balance", "power", "weighted", "optimal"])
        return case
    if kind == "learned":
        clusters = 8 * log_int(2, 128)
        return dict(kind="frame", scene="heightfield", **size(100000, 2000000), lights=log_int(2048, 16384),
                    triangles=log_int(1000, 200000), candidates=rng.randint(2, 16), frames=rng.randint(1, 4),
                    proposal=rng.choice(["learned", "learned", "clusters"]), clusters=clusters)
    if kind == "uniform":
        return dict(kind="frame", scene="heightfield", **size(30000, 500000), lights=log_int(16, 4096),
                    triangles=log_int(1000, 100000), candidates=1, frames=rng.randint(1, 4), light_sampling="uniform")
    if kind == "batch":
        lo = rng.randint(64, 300)
        return dict(kind="batch", scene="plane", items=rng.randint(2, 8), min_side=lo, max_side=lo * rng.randint(2, 4),
                    lights=log_int(32, 8192), triangles=log_int(1000, 200000), candidates=rng.randint(2, 16),
                    frames=rng.randint(1, 2))
    if kind == "logits":
        return dict(kind="logits", scene="heightfield", **size(20000, 2000000), clusters=8 * log_int(1, 64))
    if kind == "train":
        return dict(kind="train", scene="heightfield", **size(100000, 2000000), lights=log_int(2048, 16384),
                    clusters=8 * log_int(1, 128), candidates=rng.randint(4, 32), stride=rng.randint(5, 40))
    return dict(kind="rays", lights=log_int(16, 4096), triangles=log_int(1000, 300000), rays=log_int(20000, 4000000))


# ------------------------------------------------------------------ inputs --
@functools.lru_cache(maxsize=None)
def _context():
    """The program's context: one for all its scenes and frames."""
    return rl.Context(0)


def _settings(case):
    return rl.settings(candidates=case["candidates"], mis=case.get("mis", "optimal_clamped"),
                       numerics=case.get("numerics", "exact"), proposal=case.get("proposal", "uniform"),
                       light_sampling=case.get("light_sampling", "ris"), proposal_uniform_fraction=0.05,
                       shadows=case["triangles"] > 0)


def _lights(rng, count, scene):
    """std140 rows of lights facing down within 30 degrees: quads above the
    plane, jittered convex polygons of 3 to 8 vertices above the heightfield."""
    plane = scene == "plane"
    n = np.full(count, 4) if plane else rng.integers(3, 9, count)
    n[0] = 4 if plane else 8
    slot = np.arange(8)[None, :]
    angle = 2 * np.pi * (slot + (0.5 if plane else rng.uniform(-0.35, 0.35, (count, 8)))) / n[:, None]
    x, y = np.cos(angle), np.sin(angle)
    nxt = np.where(slot + 1 < n[:, None], slot + 1, 0)
    x1, y1 = np.take_along_axis(x, nxt, 1), np.take_along_axis(y, nxt, 1)
    area = 0.5 * np.sum(np.where(slot < n[:, None], x * y1 - x1 * y, 0.0), axis=1)
    want = rng.uniform(0.2, 1.0, count) ** 2 if plane else np.exp(rng.uniform(np.log(0.01), np.log(1.0), count))
    scale = np.sqrt(want / area)
    lo, hi = ((-5.0, -5.0, 1.0), (5.0, 5.0, 3.0)) if plane else ((-6.0, -6.0, 2.5), (6.0, 6.0, 4.0))
    center = rng.uniform(lo, hi, (count, 3))
    tilt = np.radians(30.0)
    a, b, c = np.pi + rng.uniform(-tilt, tilt, count), rng.uniform(-tilt, tilt, count), rng.uniform(0, 2 * np.pi, count)
    ca, sa, cb, sb, cc, sc = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(c), np.sin(c)
    u = np.stack([cc * cb, sc * cb, -sb], 1)
    v = np.stack([cc * sb * sa - sc * ca, sc * sb * sa + cc * ca, cb * sa], 1)
    normal = np.cross(v, u)  # the light model's planes face against the winding
    vert = center[:, None] + scale[:, None, None] * (x[..., None] * u[:, None] + y[..., None] * v[:, None])
    vert = np.where((slot < n[:, None])[..., None], vert, vert[:, :1])
    max_n = int(n.max())
    rows = np.zeros((count, 12 + 4 * max_n), np.float32)
    rows[:, 0:3] = np.exp(rng.uniform(np.log(0.1), np.log(10.0), (count, 3)))
    rows[:, 4:7] = normal
    rows[:, 7] = -np.sum(normal * center, axis=1)
    rows[:, 8] = n.astype(np.uint32).view(np.float32)
    rows[:, 12:].reshape(count, max_n, 4)[:, :, :3] = vert[:, :max_n]
    return rows, max_n


def _triangles(rng, count, scene):
    if not count:
        return None
    if scene == "plane":
        return rl.scenes.random_triangles(rng, count, lo=(-5.0, -5.0, 0.05), hi=(5.0, 5.0, 0.9))
    return rl.scenes.random_triangles(rng, count)


def _plane_gbuffer(width, height, seed):
    """A G-buffer on z = 0 over [-5, 5]^2 seen from (0, -6, 4)."""
    n = width * height
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.empty((17, n), dtype=torch.float32, device="cuda")
    i = torch.arange(n, device="cuda")
    g[0] = ((i % width).double() + 0.5) / width * 10.0 - 5.0
    g[1] = ((i // width).double() + 0.5) / height * 10.0 - 5.0
    g[2:5] = 0.0
    g[5] = 1.0
    view = torch.tensor([0.0, -6.0, 4.0], dtype=torch.float64, device="cuda")[:, None] - g[0:3].double()
    g[6:9] = view / view.norm(dim=0, keepdim=True)
    g[9] = g[8]
    g[10:13].uniform_(0.2, 0.8, generator=gen)
    g[13:16] = 0.02
    g[16].uniform_(0.1, 0.9, generator=gen)
    return g


def _gbuffer(case, width, height, seed):
    if case["scene"] == "plane":
        return _plane_gbuffer(width, height, seed), None
    return rl.scenes.heightfield_gbuffer_gpu(_context(), width, height, seed=seed)


def _scene(rng, lights, max_n, triangles):
    return rl.Scene(_context(), lights, max_n, *rl.scenes.synthetic_ltc(0), triangles)


def _clustered(lights, count):
    """The lights listed cluster by cluster, and the clusters' offsets."""
    order, offsets = rl.scenes.cluster_order(lights, count, seed=1, iterations=8)
    return np.ascontiguousarray(lights[order]), offsets


def _model(clusters, seed):
    """A model with the spread of outputs of a trained one."""
    model = rl.Model(_context(), clusters, seed=seed)
    params = model.get_params()
    params[FEATURES * HIDDEN + HIDDEN + HIDDEN * HIDDEN + HIDDEN:] *= 8.0
    model.set_params(params)
    model.set_input_transform(CENTER, HALF_EXTENT)
    return model, params


def _frame_inputs(case, seed):
    rng = np.random.default_rng(seed)
    lights, max_n = _lights(rng, case["lights"], case["scene"])
    offsets = None
    if case.get("clusters"):
        lights, offsets = _clustered(lights, case["clusters"])
    return rng, lights, max_n, offsets


def _batch_sides(case):
    n = case["items"]
    ratio = case["max_side"] / case["min_side"]
    return [int(round(case["min_side"] * ratio ** (k / max(n - 1, 1)))) | (k & 1) for k in range(n)]


def _train_inputs(case, seed):
    """Candidates of every pixel: lights with log-normal weights, a few of
    weight zero."""
    p, m = case["width"] * case["height"], case["candidates"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cand = torch.empty((p, m, 2), dtype=torch.int32, device="cuda")
    cand[:, :, 0] = torch.randint(0, case["lights"], (p, m), dtype=torch.int32, device="cuda", generator=gen)
    w = torch.randn((p, m), device="cuda", generator=gen).mul_(1.5).exp_()
    w *= torch.rand((p, m), device="cuda", generator=gen) > 0.05
    cand[:, :, 1] = w.view(torch.int32)
    return cand


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = dict(kind=kind, ctx=ctx, case=case, noise=seed % 100000)
    if kind == "rays":
        rng = np.random.default_rng(seed)
        lights, max_n = _lights(rng, case["lights"], "heightfield")
        s["scene"] = _scene(rng, lights, max_n, _triangles(rng, case["triangles"], "heightfield"))
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = case["rays"]
        # From points below, among and above the occluders to points on the
        # lights' level, as a light sample's shadow ray goes.
        lo, hi = torch.rand((n, 3), device="cuda", generator=gen), torch.rand((n, 3), device="cuda", generator=gen)
        lo = lo * torch.tensor([12.0, 12.0, 3.5], device="cuda") - torch.tensor([6.0, 6.0, 0.5], device="cuda")
        hi = hi * torch.tensor([12.0, 12.0, 1.5], device="cuda") - torch.tensor([6.0, 6.0, -2.5], device="cuda")
        d = hi - lo
        length = d.norm(dim=1, keepdim=True)
        rays = torch.cat([lo, torch.full((n, 1), 1e-3, device="cuda"), d / length, length - 1e-3], dim=1)
        s["rays"] = rays.contiguous()
        s["hits"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        return s
    if kind == "batch":
        rng, items = np.random.default_rng(seed), []
        for k, side in enumerate(_batch_sides(case)):
            share = (k + 1) / case["items"]
            lights, max_n = _lights(rng, max(16, int(case["lights"] * share)), "plane")
            scene = _scene(rng, lights, max_n, _triangles(rng, max(16, int(case["triangles"] * share ** 2)), "plane"))
            height = max(8, side * 9 // 16)
            p = side * height
            items.append(dict(scene=scene, gbuffer=_plane_gbuffer(side, height, seed + k), width=side, height=height,
                              settings=_settings(case), noise_seed=s["noise"] + k, frames=case["frames"],
                              out_rgb=torch.zeros((p, 3), device="cuda"),
                              reservoirs=torch.zeros((p, 4), dtype=torch.int32, device="cuda")))
        s["items"] = items
        return s
    w, h = case["width"], case["height"]
    g, prim = _gbuffer(case, w, h, seed)
    s.update(gbuffer=g, primitive=prim, width=w, height=h)
    if kind == "logits":
        s["model"], _ = _model(case["clusters"], seed)
        return s
    rng, lights, max_n, offsets = _frame_inputs(case, seed)
    s["scene"] = _scene(rng, lights, max_n, _triangles(rng, case.get("triangles", 0), case["scene"]))
    if offsets is not None:
        s["scene"].set_clusters(offsets)
        s["model"], _ = _model(case["clusters"], seed)
        s["scene"].set_model(s["model"])
    if kind == "train":
        s["model"].set_training_flags(accumulate_only=True)
        s["candidates"] = _train_inputs(case, seed)
        return s
    s["settings"] = _settings(case)
    if kind == "host":
        s["gbuffer"], s["out"] = g.cpu().numpy(), np.zeros((w * h, 3), np.float32)
        return s
    s["out"] = torch.zeros((w * h, 3), device="cuda")
    s["reservoirs"] = torch.zeros((w * h, 4), dtype=torch.int32, device="cuda")
    return s


def _frame_outputs(rgb, res):
    return dict(rgb=rgb, light=res[:, 0], w_sum=res[:, 1].view(torch.float32), p_hat=res[:, 2].view(torch.float32))


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "frame":
        rl.shade(s["ctx"], s["scene"], s["gbuffer"], s["width"], s["height"], s["settings"], noise_seed=s["noise"],
                 frames=case["frames"], out_rgb=s["out"], reservoirs=s["reservoirs"], primitive=s["primitive"])
        return _frame_outputs(s["out"], s["reservoirs"])
    if kind == "host":
        return rl.shade_host(s["ctx"], s["scene"], s["gbuffer"], s["width"], s["height"], s["settings"],
                             noise_seed=s["noise"], frames=case["frames"], out=s["out"])
    if kind == "batch":
        rl.shade_batch(s["ctx"], s["items"])
        return [_frame_outputs(it["out_rgb"], it["reservoirs"]) for it in s["items"]]
    if kind == "logits":
        return s["model"].logits(s["gbuffer"], s["width"], s["height"], primitive=s["primitive"])
    if kind == "train":
        s["model"].train(s["scene"], s["gbuffer"], s["width"], s["height"], s["candidates"], case["stride"],
                         phase=case["stride"] // 2, primitive=s["primitive"])
        return s["model"].get_gradient(clear=True)
    rl.trace_shadow(s["ctx"], s["scene"], s["rays"], s["hits"])
    return s["hits"]


# -------------------------------------------------------------------- work --
def _frame_work(pixels, case, lights, triangles, sided):
    frames = case["frames"]
    vertices = 4.0 if sided else 5.5
    # G-buffer, primitive ids, lights and triangles in; colour and reservoir out.
    nbytes = pixels * (17 * 4 + (0 if sided else 4) + 12 + (0 if case["kind"] == "host" else 16))
    nbytes += lights * (12 + 32) * 4 + triangles * 36
    per_sample = FLOPS_ESTIMATOR + (FLOPS_RAYS if triangles else 0.0)
    if case.get("light_sampling", "ris") == "ris":
        per_sample += case["candidates"] * FLOPS_VERTEX * vertices
    flops = pixels * frames * per_sample
    if case.get("proposal") == "learned":
        flops += pixels * _mlp_flops(case["clusters"])
    return nbytes, flops


def _mlp_flops(clusters):
    return 2.0 * (FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN * clusters)


def _parameters(clusters):
    return FEATURES * HIDDEN + HIDDEN + HIDDEN * HIDDEN + HIDDEN + clusters * (HIDDEN + 1)


def work(case):
    kind = case["kind"]
    if kind == "rays":
        return dict(bytes=case["rays"] * 36 + case["triangles"] * 36, flops=case["rays"] * FLOPS_RAYS)
    if kind == "batch":
        nbytes = flops = 0.0
        for k, side in enumerate(_batch_sides(case)):
            share = (k + 1) / case["items"]
            b, f = _frame_work(side * max(8, side * 9 // 16), case, max(16, int(case["lights"] * share)),
                               max(16, int(case["triangles"] * share ** 2)), True)
            nbytes, flops = nbytes + b, flops + f
        return dict(bytes=nbytes, flops=flops)
    pixels = case["width"] * case["height"]
    if kind == "logits":
        k = case["clusters"]
        return dict(bytes=pixels * (10 * 4 + 4 + 4 * k) + 4 * _parameters(k), flops=pixels * _mlp_flops(k))
    if kind == "train":
        n, k = pixels // case["stride"], case["clusters"]
        return dict(bytes=n * (10 * 4 + 4 + 8 * case["candidates"]) + 8 * _parameters(k),
                    flops=n * (3 * _mlp_flops(k) - 2.0 * FEATURES * HIDDEN))
    nbytes, flops = _frame_work(pixels, case, case["lights"], case["triangles"], case["scene"] == "plane")
    return dict(bytes=nbytes, flops=flops)


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """In 64 bits: the reservoirs' weight sums of uniformly drawn candidates,
    the logits and the training gradient.  A frame's colour, chosen light and
    p_hat have no such value: which light the reservoir keeps hangs on single
    random numbers.  Visibility is a whole number."""
    kind = case["kind"]
    if kind == "logits":
        g, prim = _gbuffer(case, case["width"], case["height"], seed)
        _, params = _model(case["clusters"], seed)
        z = torch.empty((g.shape[1], case["clusters"]), dtype=torch.float64, device="cuda")
        for at in range(0, g.shape[1], 1 << 17):
            z[at:at + (1 << 17)] = _mlp_exact(_encode(g[:, at:at + (1 << 17)]), params, case["clusters"])[-1]
        return z
    if kind == "train":
        return _gradient_exact(case, seed)
    if kind == "batch":
        rng, out = np.random.default_rng(seed), []
        for k, side in enumerate(_batch_sides(case)):
            share = (k + 1) / case["items"]
            lights, _ = _lights(rng, max(16, int(case["lights"] * share)), "plane")
            _triangles(rng, max(16, int(case["triangles"] * share ** 2)), "plane")  # advances rng as prepare() does
            height = max(8, side * 9 // 16)
            out.append(dict(rgb=None, light=None, p_hat=None, w_sum=_w_sum_exact(
                _plane_gbuffer(side, height, seed + k), None, lights, case["candidates"], seed % 100000 + k)))
        return out
    if kind != "frame" or case.get("proposal") or case.get("light_sampling"):
        return None
    g, prim = _gbuffer(case, case["width"], case["height"], seed)
    _, lights, _, _ = _frame_inputs(case, seed)
    return dict(rgb=None, light=None, p_hat=None,
                w_sum=_w_sum_exact(g, prim, lights, case["candidates"], seed % 100000))


def _encode(g):
    center = torch.tensor(CENTER, dtype=torch.float64, device="cuda")[:, None]
    u = torch.cat([(g[0:3].double() - center) / HALF_EXTENT, g[3:9].double(), g[16:17].double()], 0)
    waves = [math.pi * 2.0 ** k * u for k in range(6)]
    f = torch.stack([u] + [torch.sin(w) for w in waves] + [torch.cos(w) for w in waves], 1)  # [10, 13, P]
    return torch.nn.functional.pad(f.reshape(130, -1), (0, 0, 0, FEATURES - 130)).t()


def _mlp_layers(params, k):
    p = torch.from_numpy(np.asarray(params, np.float64)).cuda()
    w1, b1, w2, b2, w3, b3 = torch.split(p, [FEATURES * HIDDEN, HIDDEN, HIDDEN * HIDDEN, HIDDEN, k * HIDDEN, k])
    w1 = w1.view(HIDDEN, FEATURES).clone()
    w1[:, 130:] = 0.0
    return w1, b1, w2.view(HIDDEN, HIDDEN), b2, w3.view(k, HIDDEN), b3


def _mlp_exact(f, params, k):
    w1, b1, w2, b2, w3, b3 = _mlp_layers(params, k)
    h1 = torch.relu(f @ w1.t() + b1)
    h2 = torch.relu(h1 @ w2.t() + b2)
    return h1, h2, h2 @ w3.t() + b3


def _gradient_exact(case, seed):
    """Gradient of the mean cross entropy between each training pixel's
    candidate weights per cluster and softmax(logits)."""
    k, stride = case["clusters"], case["stride"]
    g, prim = _gbuffer(case, case["width"], case["height"], seed)
    _, _, _, offsets = _frame_inputs(case, seed)
    _, params = _model(k, seed)
    cluster = torch.from_numpy(np.repeat(np.arange(k), np.diff(offsets.astype(np.int64)))).cuda()
    pixels = torch.arange(stride // 2, g.shape[1], stride, device="cuda")
    cand = _train_inputs(case, seed)[pixels]
    w = cand[:, :, 1].contiguous().view(torch.float32).double()
    w1, _, w2, _, w3, _ = _mlp_layers(params, k)
    grads = [0.0] * 6
    for at in range(0, len(pixels), 1 << 15):
        part = slice(at, at + (1 << 15))
        f = _encode(g[:, pixels[part]])
        h1, h2, z = _mlp_exact(f, params, k)
        total = w[part].sum(1)
        learn = ((prim[pixels[part]] == 0) & (total > 0)).double()[:, None]
        target = torch.zeros_like(z).scatter_add_(1, cluster[cand[part, :, 0].long()], w[part])
        dz = learn * (torch.softmax(z, 1) - target / total.clamp_min(1e-300)[:, None]) / len(pixels)
        d2 = (dz @ w3) * (h2 > 0)
        d1 = (d2 @ w2) * (h1 > 0)
        g1 = d1.t() @ f
        parts = [g1, d1.sum(0), d2.t() @ h1, d2.sum(0), dz.t() @ h2, dz.sum(0)]
        grads = [a + b for a, b in zip(grads, parts)]
    return torch.cat([x.reshape(-1) for x in grads])


def _mix32(h):
    h = h ^ (h >> 16)
    h = (h * 0x85EBCA6B) & 0xFFFFFFFF
    h = h ^ (h >> 13)
    h = (h * 0xC2B2AE35) & 0xFFFFFFFF
    return h ^ (h >> 16)


def _murmur(h, k):
    k = (k * 0xCC9E2D51) & 0xFFFFFFFF
    k = ((k << 15) | (k >> 17)) & 0xFFFFFFFF
    h = h ^ ((k * 0x1B873593) & 0xFFFFFFFF)
    return ((((h << 13) | (h >> 19)) & 0xFFFFFFFF) * 5 + 0xE6546B64) & 0xFFFFFFFF


def _wang(s):
    s = ((s ^ 61) ^ (s >> 16)) * 9 & 0xFFFFFFFF
    s = ((s ^ (s >> 4)) * 0x27D4EB2D) & 0xFFFFFFFF
    return s ^ (s >> 15)


def _w_sum_exact(g, prim, lights, candidates, noise):
    """Per pixel the sum over the first frame's candidates of p_hat N, p_hat
    the length of the unshadowed LTC estimate of the light drawn."""
    np_, n = g.shape[1], lights.shape[0]
    rows = torch.from_numpy(lights).cuda().double()
    count = torch.from_numpy(lights[:, 8].copy().view(np.int32)).cuda().long()
    vert = rows[:, 12:].reshape(n, -1, 4)[:, :, :3]
    ltc0, ltc1, const = rl.scenes.synthetic_ltc(0)
    table = torch.from_numpy(np.concatenate([ltc0[0], ltc1[0]], -1)).cuda().double()
    out = torch.zeros(np_, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 21) // candidates)
    for at in range(0, np_, step):
        i = torch.arange(at, min(at + step, np_), device="cuda")
        if prim is not None:
            i = i[prim[i] == 0]
        if not len(i):
            continue
        # The drawn lights: a light draw, then a reservoir draw, per candidate.
        seed, drawn = _mix32(_murmur(_murmur(torch.zeros_like(i), i), torch.full_like(i, _wang(noise * 4)))), []
        for _ in range(candidates):
            seed = (1664525 * seed + 1013904223) & 0xFFFFFFFF
            u = seed.float() * torch.tensor(2.0 ** -32, device="cuda")
            drawn.append((u * torch.tensor(float(n), device="cuda")).long().clamp_max(n - 1))
            seed = (1664525 * seed + 1013904223) & 0xFFFFFFFF
        light = torch.stack(drawn, 1)                                  # [P, M]
        q = g[:, i].double()
        frame, to_cosine, albedo = _ltc_exact(q, table, const)
        pos, diffuse = q[0:3].t(), q[10:13].t()
        rel = vert[light] - pos[:, None, None, :]                      # [P, M, V, 3]
        v = torch.einsum("pab,pmvb->pmva", frame, rel)
        plane = rows[light][:, :, 4:8]
        flip = (torch.einsum("pmk,pk->pm", plane[:, :, :3], pos) + plane[:, :, 3]) < 0
        v[..., 1] = torch.where(flip[..., None], -v[..., 1], v[..., 1])
        c = torch.einsum("pab,pmvb->pmva", to_cosine, v)
        k = count[light]
        cd, cs = _integral_exact(v, k), _integral_exact(c, k)
        color = (cd[..., None] * diffuse[:, None] + (cs * albedo[:, None])[..., None]) * rows[light][:, :, 0:3]
        out[i] = color.norm(dim=-1).sum(1) * n
    return out


def _ltc_exact(q, table, const):
    """World-to-shading rotation, shading-to-cosine matrix and albedo."""
    normal, view = q[3:6], q[6:9]
    height, width = table.shape[:2]
    cos = (normal * view).sum(0)
    tx = q[16].clamp(0, 1).sqrt() * float(const[2]) + float(const[3])
    ty = torch.acos(cos.clamp(0, 1)) * float(const[4]) + float(const[5])
    fx, fy = tx * width - 0.5, ty * height - 0.5
    x0, y0 = fx.floor(), fy.floor()
    ax, ay = (fx - x0)[:, None], (fy - y0)[:, None]
    xi = [(x0.long() + k).clamp(0, width - 1) for k in (0, 1)]
    yi = [(y0.long() + k).clamp(0, height - 1) for k in (0, 1)]
    top = table[yi[0], xi[0]] * (1 - ax) + table[yi[0], xi[1]] * ax
    bottom = table[yi[1], xi[0]] * (1 - ax) + table[yi[1], xi[1]] * ax
    t = top * (1 - ay) + bottom * ay
    x_axis = view - cos * normal
    x_axis = x_axis / x_axis.norm(dim=0, keepdim=True)
    y_axis = torch.cross(normal, x_axis, dim=0)
    frame = torch.stack([x_axis.t(), y_axis.t(), normal.t()], 1)
    zero = torch.zeros_like(cos)
    to_cosine = torch.stack([torch.stack([t[:, 0], zero, t[:, 3]], 1), torch.stack([zero, t[:, 2], zero], 1),
                             torch.stack([-t[:, 1], zero, t[:, 4]], 1)], 1)
    return frame, to_cosine, t[:, 5]


def _edge_exact(a, b):
    a, b = a / a.norm(dim=-1, keepdim=True), b / b.norm(dim=-1, keepdim=True)
    x = (a * b).sum(-1)
    y = x.abs()
    v = (0.8543985 + (0.4965155 + 0.0145206 * y) * y) / (3.4175940 + (4.1616724 + y) * y)
    v = torch.where(x > 0, v, 0.5 / (1 - x * x).clamp_min(1e-7).sqrt() - v)
    return (a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]) * v


def _integral_exact(v, count):
    """|sum of the edge integrals| of the polygon's part above z = 0."""
    slots = v.shape[-2]
    total = torch.zeros_like(v[..., 0, 0])
    leave = torch.ones_like(v[..., 0, :])
    enter = torch.ones_like(leave)
    crosses = torch.zeros_like(total, dtype=torch.bool)
    for j in range(slots):
        used = j < count
        b = torch.where((j + 1 < count)[..., None], v[..., min(j + 1, slots - 1), :], v[..., 0, :])
        a = v[..., j, :]
        above_a, above_b = a[..., 2] > 0, b[..., 2] > 0
        dz = a[..., 2] - b[..., 2]
        cut = a + (a[..., 2] / torch.where(dz == 0, torch.ones_like(dz), dz))[..., None] * (b - a)
        cut = torch.cat([cut[..., :2], torch.zeros_like(cut[..., 2:])], -1)
        out, into = used & above_a & ~above_b, used & ~above_a & above_b
        leave, enter = torch.where(out[..., None], cut, leave), torch.where(into[..., None], cut, enter)
        crosses |= out
        total += torch.where(used & (above_a | above_b), _edge_exact(torch.where(into[..., None], cut, a),
                                                                     torch.where(out[..., None], cut, b)), 0.0)
    return (total + torch.where(crosses, _edge_exact(leave, enter), 0.0)).abs()
