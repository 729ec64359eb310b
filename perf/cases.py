"""The workloads on which the denoiser's speed is followed: whole frames and
clips through a plan, the five drop-in stages, the fitter alone and steps of
the many-stream engine, from the smallest images that a plan accepts up to
3840x2160.

Inputs are rendered by the repository's seeded scene source (ground plane and
spheres, 1-sample noise with fireflies), as in its benchmark and tests.  A
pass of a plan or a batch starts its streams anew (frame 0) and denoises
`frames` consecutive frames, so that equal inputs give equal outputs; all
frames but the first take history.
"""
import torch

import bmfr_b200 as bmfr
from bmfr_scene import Scene

BLOCK_OFFSETS = ((-14, -14), (4, -6), (-8, 14), (8, 0), (-10, -8), (2, 12), (12, -12), (-10, 0),
                 (12, 14), (-8, -16), (6, 6), (-2, -2), (6, -14), (-16, 12), (14, -4), (-6, 4))
PRECISION = {"qr": bmfr.QR_CHOLESKY2, "half_history": 1}


def listed():
    return [
        # An application's smallest viewport, a call per frame: launches and latency.
        {"name": "frames_64x48", "kind": "frames", "width": 64, "height": 48, "frames": 4},
        # A preview window of odd size in the precision form, a call per frame.
        {"name": "frames_427x241_precision", "kind": "frames", "width": 427, "height": 241, "frames": 4, **PRECISION},
        # The interactive renderer at the reference's own resolution: one call for each frame.
        {"name": "frames_1280x720", "kind": "frames", "width": 1280, "height": 720, "frames": 4},
        # A recorded camera path at that resolution: all its frames in one call.
        {"name": "clip_1280x720", "kind": "clip", "width": 1280, "height": 720, "frames": 8},
        # float32 tmp_data, the reference's other compile-time choice, at a size no tile divides.
        {"name": "clip_853x481_f32", "kind": "clip", "width": 853, "height": 481, "frames": 4, "half_tmp": 0},
        # The fused pipeline, for callers that have no room for tmp_data, at a ragged size.
        {"name": "frames_1277x717_fused", "kind": "frames", "width": 1277, "height": 717, "frames": 4, "fused": 1},
        # Full HD in the precision form.
        {"name": "clip_1920x1080_precision", "kind": "clip", "width": 1920, "height": 1080, "frames": 4, **PRECISION},
        # The largest frames in use, reference arithmetic.
        {"name": "clip_3840x2160", "kind": "clip", "width": 3840, "height": 2160, "frames": 4},
        # A host loop moved over from the reference: its five kernels, one call each.
        {"name": "stages_1280x720", "kind": "stages", "width": 1280, "height": 720},
        # The fit alone, for renderers with features and filters of their own.
        {"name": "fitter_1280x720", "kind": "fitter", "width": 1280, "height": 720},
        {"name": "fitter_1920x1080_precision", "kind": "fitter", "width": 1920, "height": 1080,
         "qr": bmfr.QR_CHOLESKY2},
        # A render server's step over viewers of different sizes (the engine's usual parameters).
        {"name": "batch_8_streams", "kind": "batch", "frames": 2, **PRECISION,
         "sizes": "640x360,640x360,640x360,1280x720,1280x720,1280x720,1920x1080,1920x1080"},
    ]


def _side(rng, low, high):
    """A side spread over the logarithm of [low, high], of either parity, that a plan accepts."""
    while True:
        n = round(low * (high / low) ** rng.random())
        if 32 * -(-n // 32) + 30 <= 2 * n:   # the mirrored margin stays within one image
            return n


def draw(rng):
    kind = rng.choice(("frames", "frames", "clip", "clip", "stages", "fitter", "batch"))
    if kind == "batch":
        sizes = []
        for _ in range(rng.randint(2, 8)):
            w = _side(rng, 96, 1920)
            sizes.append("%dx%d" % (w, _side(rng, max(47, w // 3), max(64, w * 9 // 16))))
        return {"kind": kind, "frames": 2, "sizes": ",".join(sizes), **(PRECISION if rng.random() < 0.7 else {})}
    w = _side(rng, 32, 3840)
    case = {"kind": kind, "width": w, "height": _side(rng, max(32, w // 3), max(47, w * 9 // 16))}
    if kind in ("frames", "clip"):
        case["frames"] = rng.choice((2, 4))
    form = rng.random()
    if kind != "stages" and form < 0.35:
        case.update(PRECISION if kind != "fitter" else {"qr": bmfr.QR_CHOLESKY2})
    elif form < 0.5 and w <= 1920:
        case["half_tmp"] = 0
    elif kind == "frames" and form < 0.65:
        case["fused"] = 1
    return case


def _params(case, scene):
    return bmfr.default_params(position_limit_squared=scene.position_limit_squared,
                               normal_limit_squared=scene.normal_limit_squared,
                               use_half_precision_in_tmp_data=case.get("half_tmp", 1), fp32_qr=case.get("qr", 0),
                               half_history=case.get("half_history", 0),
                               pipeline=bmfr.PIPELINE_FUSED if case.get("fused") else bmfr.PIPELINE_STAGED)


def _render(seed, width, height, frames):
    """The scene and `frames` rendered frames of it, as dicts of (height, width, 3) tensors."""
    scene = Scene(seed, width, height, 12)
    got = []
    for f in range(frames):
        d = {k: torch.empty(height, width, 3, device="cuda") for k in ("albedo", "normals", "positions", "noisy", "clean")}
        scene.render_device(f, **d)
        d["matrix"], d["offset"] = scene.prev_camera(f), scene.pixel_offset(f)
        got.append(d)
    return scene, got


def _io(frames, f, result):
    """The buffers of frame f: its own, the previous frame's normals and positions, where the result goes."""
    now, before = frames[f], frames[f - 1] if f else {}
    return {**{k: now[k] for k in ("albedo", "normals", "positions", "noisy")}, "result": result,
            "previous_normals": before.get("normals"), "previous_positions": before.get("positions")}


class _Device:
    """Device memory of a plan as something torch can view; a view keeps the plan."""

    def __init__(self, plan, pointer, shape, kind):
        self.plan = plan
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "typestr": kind, "version": 3}


def _history(plan, half):
    """What the frame after an even number of frames starts from, as views of the plan's buffers."""
    b, shape, kind = plan.buffers(), (plan.height, plan.width, 3), "<f2" if half else "<f4"
    views = {"noisy": (b.accumulated_noisy, shape, kind), "filtered": (b.accumulated_filtered, shape, kind),
             "spp": (b.spp, shape[:2], "|u1")}
    return {k: torch.as_tensor(_Device(plan, *v), device="cuda") for k, v in views.items()}


def _sizes(case):
    return [tuple(int(n) for n in s.split("x")) for s in case["sizes"].split(",")]


def _stage_inputs(case, seed):
    """Frame 1 of a scene with frame 0's outputs in a form that needs no denoiser: the raw frame as the
    accumulated colour, any sample counts, and the noise-free image as the filtered and displayed ones."""
    scene, frames = _render(seed, case["width"], case["height"], 2)
    gen = torch.Generator("cuda").manual_seed(seed)
    clean, shape = frames[0]["clean"], frames[0]["clean"].shape[:2]
    return scene, frames, {"noisy": frames[0]["noisy"], "filtered": clean,
                           "spp": torch.randint(1, 30, shape, generator=gen, device="cuda", dtype=torch.uint8),
                           "result": (clean * frames[0]["albedo"]).clamp(0, 1).sqrt()}


def _features(frame, colour, number):
    """The 13 columns of every 32x32 block of the margin grid of frame `number`: [blocks, 1024, 13]."""
    h, w = frame["positions"].shape[:2]
    bx, by = -(-w // 32) + 1, -(-h // 32) + 1
    ox, oy = BLOCK_OFFSETS[number % 16]

    def mirrored(n, blocks, offset):
        i = torch.arange(32 * blocks, device=colour.device) - 16 + offset
        return torch.where(i < 0, -i - 1, torch.where(i >= n, 2 * n - i - 1, i))

    y, x = mirrored(h, by, oy)[:, None], mirrored(w, bx, ox)[None, :]
    n, p, c = (t.to(colour.dtype)[y, x] for t in (frame["normals"], frame["positions"], colour))
    t = torch.cat((torch.ones_like(n[..., :1]), n, p, p * p, c), -1)
    return t.reshape(by, 32, bx, 32, 13).permute(0, 2, 1, 3, 4).reshape(by * bx, 1024, 13)


def _tmp(features, half):
    return features.transpose(1, 2).contiguous().to(torch.float16 if half else torch.float32)


def prepare(case, seed):
    kind, half_tmp = case["kind"], bool(case.get("half_tmp", 1))
    if kind == "batch":
        streams, slots, ios = [], [], []
        batch = None
        for k, (w, h) in enumerate(_sizes(case)):
            scene, frames = _render(seed + 101 * k, w, h, case["frames"])
            batch = batch or bmfr.Batch(_params(case, scene))
            slots.append(batch.add_stream(w, h))
            streams.append((frames, [torch.empty(h, w, 3, device="cuda") for _ in frames]))
        for f in range(case["frames"]):
            ios.append(([bmfr.Batch.frame_io(**_io(fr, f, out[f])) for fr, out in streams],
                        [fr[f]["matrix"] for fr, _ in streams], [fr[f]["offset"] for fr, _ in streams]))
        return {"kind": kind, "batch": batch, "slots": slots, "ios": ios, "streams": streams}
    w, h = case["width"], case["height"]
    if kind in ("frames", "clip"):
        scene, frames = _render(seed, w, h, case["frames"])
        plan = bmfr.Plan(w, h, _params(case, scene))
        results = [torch.empty(h, w, 3, device="cuda") for _ in frames]
        return {"kind": kind, "plan": plan, "frames": [_io(frames, f, r) for f, r in enumerate(results)],
                "matrices": [f["matrix"] for f in frames], "offsets": [f["offset"] for f in frames],
                "out": {"frames": results, "history": _history(plan, case.get("half_history"))}}
    scene, frames, before = _stage_inputs(case, seed)
    plan = bmfr.Plan(w, h, _params(case, scene))
    blocks = plan.sizes.blocks
    tmp = _tmp(_features(frames[1], frames[1]["noisy"], 1), half_tmp)
    out = {"weights": torch.empty(blocks, 10, 3, device="cuda"), "bounds": torch.empty(blocks, 6, 2, device="cuda")}
    if kind == "stages":
        out.update({k: torch.empty(h, w, 3, device="cuda") for k in ("noisy", "filtered", "accumulated", "mapped", "result")})
        out.update({k: torch.empty(h, w, dtype=torch.uint8, device="cuda") for k in ("accept", "spp")})
        out.update(pixel=torch.empty(h, w, 2, device="cuda"), tmp=torch.empty_like(tmp))
    return {"kind": kind, "plan": plan, "now": frames[1], "last": frames[0], "before": before, "tmp": tmp, "out": out}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        batch, slots = state["batch"], state["slots"]
        for s in slots:
            batch.reset_stream(s)
        for io, matrices, offsets in state["ios"]:
            batch.step(slots, matrices, offsets, io)
        return [out for _, out in state["streams"]]
    plan, out = state["plan"], state["out"]
    if kind == "clip":
        plan.reset()
        plan.denoise_frames(state["frames"], state["matrices"], state["offsets"])
    elif kind == "frames":
        plan.reset()
        for io, matrix, offset in zip(state["frames"], state["matrices"], state["offsets"]):
            plan.denoise_frame_io(prev_frame_camera_matrix=matrix, pixel_offset=offset, **io)
    elif kind == "fitter":
        bmfr.fitter(plan, out["weights"], out["bounds"], state["tmp"], 1)
    else:
        now, last, before = state["now"], state["last"], state["before"]
        out["noisy"].copy_(now["noisy"])   # the frame's colour arrives in the buffer that is blended in place
        bmfr.accumulate_noisy_data(plan, out["pixel"], out["accept"], now["normals"], last["normals"], now["positions"],
                                   last["positions"], out["noisy"], before["noisy"], before["spp"], out["spp"],
                                   out["tmp"], now["matrix"], now["offset"], 1)
        bmfr.fitter(plan, out["weights"], out["bounds"], out["tmp"], 1)
        bmfr.weighted_sum(plan, out["weights"], out["bounds"], out["filtered"], now["normals"], now["positions"],
                          out["noisy"], 1)
        bmfr.accumulate_filtered_data(plan, out["filtered"], out["pixel"], out["accept"], now["albedo"], out["mapped"],
                                      out["spp"], before["filtered"], out["accumulated"], 1)
        bmfr.taa(plan, out["pixel"], out["mapped"], out["result"], before["result"], 1)
    return out


def work(case):
    if case["kind"] == "batch":
        each = [work({**case, "kind": "frames", "width": w, "height": h}) for w, h in _sizes(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    w, h, tmp, colour = case["width"], case["height"], 2 if case.get("half_tmp", 1) else 4, 6 if case.get("half_history") else 12
    blocks, pixels = (-(-w // 32) + 1) * (-(-h // 32) + 1), w * h
    # Ten reflections of a 1024-row block, 12 to 3 columns after each: a product and an update of 2 operations each.
    fit = blocks * 4 * 1024 * 75
    if case["kind"] == "fitter":
        return {"bytes": blocks * (13 * 1024 * tmp + 42 * 4), "flops": fit}
    if case["kind"] == "stages":
        # Frame, last frame's normals, positions and three histories in; the stages' buffers out.
        return {"bytes": pixels * (48 + 24 + 37 + 12 * 5 + 10) + blocks * (13 * 1024 * tmp + 42 * 4), "flops": fit + 400 * pixels}
    # Four inputs, the previous normals and positions, the result; the three histories and the sample counts both ways.
    history = 2 * (3 * colour + 1)
    return {"bytes": case["frames"] * pixels * (48 + 24 + 12 + history) - pixels * (24 + history // 2),
            "flops": case["frames"] * (fit + 400 * pixels)}


# ---- the same results in 64 bits -------------------------------------------

def _noise(rows, number):
    """random(i) - 0.5 of features 1..9 (opencl/bmfr.cl:162-182): [rows, 9]."""
    i = torch.arange(rows, device="cuda")[:, None] + 1024 * torch.arange(1, 10, device="cuda") + number * 13 * 1024
    m = 0xffffffff
    a = ((i + 0x7ed55d16) + (i << 12)) & m
    a = (a ^ 0xc761c23c) ^ (a >> 19)
    a = ((a + 0x165667b1) + (a << 5)) & m
    a = ((a + 0xd3a2646c) & m) ^ ((a << 9) & m)
    a = ((a + 0xfd7046c5) + (a << 3)) & m
    a = (a ^ 0xb55a4f09) ^ (a >> 16)
    return a.double() / 4294967296.0 - 0.5


def _scaled(v, bounds):
    """Features 4..9 scaled by their block's bounds (opencl/bmfr.cl:200-205)."""
    low, d = bounds[..., 0], bounds[..., 1] - bounds[..., 0]
    return torch.where(d.abs() > 1, (v - low) / d, v - low)


def _fit64(features, number):
    """Least squares of the three colours on the ten features of each block: weights and bounds."""
    a, b = features[..., :10].clone(), features[..., 10:]
    v = a[..., 4:]
    bounds = torch.stack((v.amin(1), v.amax(1)), -1)
    a[..., 4:] = _scaled(v, bounds[:, None])
    a[..., 1:] += 0.02 * _noise(1024, number)
    r = torch.eye(10, dtype=a.dtype, device=a.device).expand(a.shape[0], 10, 10)
    q = a
    for _ in range(2):   # CholeskyQR, twice: orthogonal to 64 bits for these condition numbers
        upper = torch.linalg.cholesky(q.transpose(1, 2) @ q).transpose(1, 2)
        q = torch.linalg.solve_triangular(upper, q, upper=True, left=False)
        r = upper @ r
    return torch.linalg.solve_triangular(r, q.transpose(1, 2) @ b, upper=True), bounds


def _taps(pixel, h, w):
    """The four bilinear taps of each position: (index, weight, inside the image)."""
    pixel = torch.nan_to_num(pixel, 1e9, 1e9, -1e9).clamp(-1e9, 1e9)
    low = pixel.floor()
    f, low = pixel - low, low.long()
    for k in range(4):
        dx, dy = k & 1, k >> 1
        x, y = low[..., 0] + dx, low[..., 1] + dy
        weight = (f[..., 0] if dx else 1 - f[..., 0]) * (f[..., 1] if dy else 1 - f[..., 1])
        yield y.clamp(0, h - 1) * w + x.clamp(0, w - 1), weight, (x >= 0) & (y >= 0) & (x < w) & (y < h)


def _accumulate64(frame, last, noisy, spp, limits):
    """accumulate_noisy_data: blended colour, sample counts, reprojected positions, accepted taps."""
    h, w = noisy.shape[:2]
    p, n, colour = (frame[k].double() for k in ("positions", "normals", "noisy"))
    m = torch.as_tensor(frame["matrix"], device="cuda").double().reshape(4, 4)
    off = torch.as_tensor(frame["offset"], device="cuda").double()
    q = p @ m[:3] + m[3]
    size = torch.tensor([w, h], dtype=torch.float64, device="cuda")
    pixel = (q[..., :2] / q[..., 3:] + 1) / 2 * size - torch.stack((off[0], 1 - off[1]))
    total, previous, samples, accept = torch.zeros_like(p[..., 0]), torch.zeros_like(p), torch.zeros_like(p[..., 0]), []
    lp, ln, lc, ls = (t.double().reshape(h * w, -1) for t in (last["positions"], last["normals"], noisy, spp))
    for i, weight, inside in _taps(pixel, h, w):
        ok = inside & (((lp[i] - p) ** 2).sum(-1) < limits[0]) & (((ln[i] - n) ** 2).sum(-1) < limits[1])
        weight = torch.where(ok, weight, 0.0)
        total, previous = total + weight, previous + weight[..., None] * lc[i]
        samples = samples + weight * ls[i][..., 0]
        accept.append(ok)
    some = total > 0
    total = torch.where(some, total, 1.0)
    previous, samples = previous / total[..., None], samples / total
    alpha = torch.where(some, (1 / (samples + 1)).clamp(min=0.2), 1.0)[..., None]
    counts = torch.where(alpha[..., 0] < 1, (samples.round() + 1).clamp(max=255), 1.0)
    return alpha * colour + (1 - alpha) * previous, counts, pixel, accept


def _weighted_sum64(frame, weights, bounds, number):
    h, w = frame["positions"].shape[:2]
    ox, oy = BLOCK_OFFSETS[number % 16]
    x = (torch.arange(w, device="cuda") + 16 - ox) // 32
    y = (torch.arange(h, device="cuda") + 16 - oy) // 32
    block = y[:, None] * (-(-w // 32) + 1) + x[None, :]
    n, p = frame["normals"].double(), frame["positions"].double()
    got = weights[:, 0][block]
    v = torch.cat((p, p * p), -1)
    for k in range(3):
        got = got + weights[:, 1 + k][block] * n[..., k:k + 1]
    for k in range(6):
        got = got + weights[:, 4 + k][block] * _scaled(v[..., k], bounds[:, k][block])[..., None]
    return got.clamp(min=0)


def _accumulate_filtered64(filtered, pixel, accept, counts, before, albedo):
    """accumulate_filtered_data: accumulated and tone-mapped colours."""
    h, w = filtered.shape[:2]
    alpha, previous = torch.ones_like(filtered[..., :1]), torch.zeros_like(filtered)
    if before is not None:
        total = torch.zeros_like(filtered[..., 0])
        for (i, weight, _), ok in zip(_taps(pixel, h, w), accept):
            weight = torch.where(ok, weight, 0.0)
            total, previous = total + weight, previous + weight[..., None] * before.double().reshape(-1, 3)[i]
        some = (total > 0)[..., None]
        previous = torch.where(some, previous / total[..., None], previous)
        alpha = torch.where(some, (1 / counts).clamp(min=0.1)[..., None], 1.0)
    got = alpha * filtered + (1 - alpha) * previous
    return got, (got * albedo.double()).clamp(min=0).pow(0.454545).clamp(0, 1)


def _taa64(pixel, new, before):
    h, w = new.shape[:2]
    to = torch.tensor([[1, 2, 1], [2, 0, -2], [-1, 2, -1]], dtype=torch.float64, device="cuda")
    back = torch.tensor([[1, 1, -1], [1, 0, 1], [1, -1, -1]], dtype=torch.float64, device="cuda") / 4
    ycc = new @ to.T
    edges = []
    for sign in (1, -1):   # the largest of the 3x3 box and of the cross, then the smallest
        t = torch.nn.functional.pad((sign * ycc).permute(2, 0, 1), (1, 1, 1, 1), value=-float("inf"))
        at = [[t[:, y:y + h, x:x + w] for x in range(3)] for y in range(3)]
        cross = torch.stack((at[0][1], at[1][0], at[1][1], at[1][2], at[2][1])).amax(0)
        corners = torch.stack((at[0][0], at[0][2], at[2][0], at[2][2])).amax(0)
        edges.append(sign * ((cross + torch.maximum(cross, corners)) / 2).permute(1, 2, 0))
    total, previous = torch.zeros_like(new[..., 0]), torch.zeros_like(new)
    for i, weight, inside in _taps(pixel, h, w):
        weight = torch.where(inside, weight, 0.0)
        total, previous = total + weight, previous + weight[..., None] * before.double().reshape(-1, 3)[i]
    clamped = torch.minimum(torch.maximum((previous / total[..., None]) @ to.T, edges[1]), edges[0])
    low = torch.nan_to_num(pixel, 1e9, 1e9, -1e9).floor()
    seen = (low >= -1).all(-1) & (low[..., 0] < w) & (low[..., 1] < h)
    return torch.where(seen[..., None], 0.2 * new + 0.8 * (clamped @ back.T), new)


def _clip64(scene, frames):
    """Every frame's result, and the histories after the last."""
    limits, got = (scene.position_limit_squared, scene.normal_limit_squared), []
    noisy = filtered = counts = None
    for f, frame in enumerate(frames):
        if f:
            noisy, counts, pixel, accept = _accumulate64(frame, frames[f - 1], noisy, counts, limits)
        else:
            noisy, pixel, accept = frame["noisy"].double(), None, None
            counts = torch.ones_like(noisy[..., 0])
        weights, bounds = _fit64(_features(frame, noisy, f), f)
        now = _weighted_sum64(frame, weights, bounds, f)
        filtered, mapped = _accumulate_filtered64(now, pixel, accept, counts, filtered, frame["albedo"])
        got.append(_taa64(pixel, mapped, got[-1]) if f else mapped)
    return {"frames": got, "history": {"noisy": noisy, "filtered": filtered, "spp": None}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_clip64(*_render(seed + 101 * k, w, h, case["frames"]))["frames"] for k, (w, h) in enumerate(_sizes(case))]
    if kind in ("frames", "clip"):
        return _clip64(*_render(seed, case["width"], case["height"], case["frames"]))
    # The reference's arithmetic rounds the system to 16 bits after every reflection: its weights have no value in
    # 64 bits (those of nearly dependent features are of any size), what is computed from them has.
    scene, frames, before = _stage_inputs(case, seed)
    now = frames[1]
    if kind == "fitter":
        tmp = _tmp(_features(now, now["noisy"], 1), bool(case.get("half_tmp", 1)))
        weights, bounds = _fit64(tmp.double().transpose(1, 2), 1)
        return {"weights": weights if case.get("qr") else None, "bounds": bounds}
    limits = (scene.position_limit_squared, scene.normal_limit_squared)
    noisy, counts, pixel, accept = _accumulate64(now, frames[0], before["noisy"], before["spp"], limits)
    features = _features(now, noisy, 1)
    weights, bounds = _fit64(features, 1)
    filtered = _weighted_sum64(now, weights, bounds, 1)
    accumulated, mapped = _accumulate_filtered64(filtered, pixel, accept, counts, before["filtered"], now["albedo"])
    return {"weights": None, "bounds": bounds, "noisy": noisy, "filtered": filtered, "accumulated": accumulated,
            "mapped": mapped, "result": _taa64(pixel, mapped, before["result"]), "accept": None, "spp": None,
            "pixel": pixel, "tmp": features.transpose(1, 2)}
