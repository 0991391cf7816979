"""Performance cases: the calls a user of imageproc_b200 makes, with their
inputs, one pass of each, the work of a pass and the exact results.

A case is a dict of plain values whose "kind" names the call. Sizes are those
of the benchmark, the tests and the tools that ship with the package, odd and
ragged ones among them; `draw` gives more cases of the same ranges.
"""

import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from imageproc_b200 import _lib, device, learned
from imageproc_b200 import template_matching as tm

SSE, SSE_NORM, CCORR, CCORR_NORM = 0, 1, 2, 3
U8, I16, F32 = 0, 5, 8    # ipb_elem_type codes of filter outputs
NET_LAYERS = (1, 32, 32, 32, 32)  # input channels of the proposal network's convolutions


def listed():
    return [
        # a tracker's or a UI test's search in a small window: latency and launches count
        {"name": "map_512_t16", "kind": "map", "W": 512, "H": 512, "w": 16, "h": 16, "method": SSE, "mask": 0,
         "extremes": False, "content": "uniform"},
        # find one template in a full-HD frame: the score map, then its extremes on the host
        {"name": "locate_1080p_t64", "kind": "map", "W": 1920, "H": 1080, "w": 64, "h": 64, "method": CCORR_NORM,
         "mask": 0, "extremes": True, "content": "blobs"},
        # an irregular part searched with a binary mask, every size odd
        {"name": "masked_1283x957_t57x43", "kind": "map", "W": 1283, "H": 957, "w": 57, "h": 43,
         "method": SSE_NORM, "mask": 1, "extremes": False, "content": "blobs"},
        # the drop-in call with host arrays, copies and all
        {"name": "host_1080p_t64", "kind": "host_map", "W": 1920, "H": 1080, "w": 64, "h": 64, "method": SSE,
         "content": "blobs"},
        # every method, unmasked and masked, of one frame in one planned batch (the benchmark's step)
        {"name": "plan_eight_maps_1080p", "kind": "eight", "W": 1920, "H": 1080, "w": 64, "h": 64},
        # a serving batch of unrelated images and templates of every size
        {"name": "plan_uneven_60", "kind": "uneven", "n": 60, "lo": 256, "hi": 4096, "tmin": 8, "tmax": 128},
        # a template library against one image, scores and best positions
        {"name": "many_2048_n128_t32", "kind": "many", "W": 2048, "H": 2048, "n": 128, "w": 32, "h": 32,
         "method": CCORR_NORM},
        # 64 queries on a large scene through the learned proposals
        {"name": "propose_8192_n64", "kind": "propose", "side": 8192, "n": 64},
        # training the proposal network: forward and backward of one batch
        {"name": "net_gradients_b128", "kind": "gradients", "n": 128, "crop": 96},
        # peaks of a score map
        {"name": "suppress_4065_r8", "kind": "suppress", "W": 4065, "H": 4065, "r": 8},
        # box statistics of a large image
        {"name": "integral_sq_u64_4096", "kind": "integral", "W": 4096, "H": 4096, "channels": 1, "bits": 64,
         "squared": True},
        # smoothing an image before matching
        {"name": "filter_5x5_4096", "kind": "filter", "W": 4096, "H": 4096, "channels": 1, "kw": 5, "kh": 5,
         "float": True, "out": U8},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["map", "map", "map", "host_map", "eight", "uneven", "many", "propose", "gradients",
                       "suppress", "integral", "filter"])
    if kind in ("map", "host_map", "eight"):
        w, h = rng.randint(5, 128), rng.randint(5, 128)
        c = {"kind": kind, "W": _log_uniform(rng, 256, 2560), "H": _log_uniform(rng, 256, 2160), "w": w, "h": h}
        if kind == "eight":
            return dict(c, w=max(w, 8), h=max(h, 8))
        c.update(method=rng.randrange(4), content=rng.choice(["uniform", "blobs"]))
        if kind == "map":
            c.update(mask=rng.choice([0, 0, 1]), extremes=rng.random() < 0.5)
        return c
    if kind == "uneven":
        return {"kind": kind, "n": _log_uniform(rng, 4, 56), "lo": 256, "hi": rng.randint(1024, 4096), "tmin": 8,
                "tmax": rng.randint(24, 128)}
    if kind == "many":
        return {"kind": kind, "W": _log_uniform(rng, 256, 2048), "H": _log_uniform(rng, 256, 2048),
                "n": _log_uniform(rng, 8, 128), "w": rng.randint(16, 48), "h": rng.randint(8, 48),
                "method": rng.randrange(4)}
    if kind == "propose":
        return {"kind": kind, "side": 32 * rng.randint(64, 250), "n": _log_uniform(rng, 4, 64)}
    if kind == "gradients":
        return {"kind": kind, "n": _log_uniform(rng, 16, 127), "crop": 96}
    W, H = _log_uniform(rng, 256, 4096), _log_uniform(rng, 256, 4096)
    if kind == "suppress":
        return {"kind": kind, "W": W, "H": H, "r": rng.randint(1, 16)}
    if kind == "integral":
        return {"kind": kind, "W": W, "H": H, "channels": rng.choice([1, 1, 3]), "bits": rng.choice([32, 64]),
                "squared": rng.random() < 0.5}
    is_float = rng.random() < 0.7
    return {"kind": kind, "W": W, "H": H, "channels": rng.choice([1, 1, 3]), "kw": rng.randint(1, 7),
            "kh": rng.randint(1, 7), "float": is_float, "out": rng.choice([U8, F32]) if is_float else I16}


# ---- inputs ---------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform_u8(shape, g):
    return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)


def _blobs(W, H, g):
    """200 isotropic Gaussian blobs plus noise in [-8, 8]."""
    r = torch.rand((4, 200), generator=g, device="cuda")
    cx, cy, sigma, amp = r[0] * W, r[1] * H, 5 + 75 * r[2], 20 + 180 * r[3]
    xs, ys = torch.arange(W, device="cuda"), torch.arange(H, device="cuda")
    gx = torch.exp(-0.5 * ((xs[None] - cx[:, None]) / sigma[:, None]) ** 2)
    gy = amp[:, None] * torch.exp(-0.5 * ((ys[None] - cy[:, None]) / sigma[:, None]) ** 2)
    noise = torch.randint(-8, 9, (H, W), generator=g, device="cuda")
    return (gy.T @ gx + noise).round().clamp(0, 255).to(torch.uint8)


def _value_noise(W, H, g):
    """Three octaves of value noise (lattices of 64, 16 and 4 pixels)."""
    acc = torch.zeros((H, W), device="cuda")
    for lattice, weight in ((64, 0.6), (16, 0.3), (4, 0.1)):
        grid = torch.rand((H // lattice + 2, W // lattice + 2), generator=g, device="cuda")

        def axis(n):
            f = torch.arange(n, device="cuda") / lattice
            i = f.long()
            t = f - i
            return i, t * t * (3 - 2 * t)

        (iy, sy), (ix, sx) = axis(H), axis(W)
        rows = grid[iy] + (grid[iy + 1] - grid[iy]) * sy[:, None]
        acc += weight * (rows[:, ix] + (rows[:, ix + 1] - rows[:, ix]) * sx[None])
    return (acc * 255).round().clamp(0, 255).to(torch.uint8)


def _crops(image, n, w, h, g, brightness, noise):
    """n crops of the image with a brightness offset and per-pixel noise."""
    H, W = image.shape
    ys = torch.randint(0, H - h + 1, (n,), generator=g, device="cuda")
    xs = torch.randint(0, W - w + 1, (n,), generator=g, device="cuda")
    rows = ys[:, None] + torch.arange(h, device="cuda")
    cols = xs[:, None] + torch.arange(w, device="cuda")
    t = image[rows[:, :, None], cols[:, None, :]].int()
    if brightness:
        t = t + torch.randint(-brightness, brightness + 1, (n, 1, 1), generator=g, device="cuda", dtype=torch.int32)
    t = t + torch.randint(-noise, noise + 1, t.shape, generator=g, device="cuda", dtype=torch.int32)
    return t.clamp(0, 255).to(torch.uint8)


def _match_inputs(case, seed):
    g = _gen(seed)
    W, H, w, h = case["W"], case["H"], case["w"], case["h"]
    if case.get("content") == "uniform":
        image = _uniform_u8((H, W), g)
        template = _crops(image, 1, w, h, g, 0, 4)[0]
    else:
        image = _blobs(W, H, g)
        template = _crops(image, 1, w, h, g, 10, 0)[0]
    mask = (torch.rand((h, w), generator=g, device="cuda") < 0.8).to(torch.uint8)
    return image, template.contiguous(), mask


def _eight_items(case, seed):
    image, template, mask = _match_inputs(case, seed)
    return [(image, template, m) for m in range(4)] + [(image, template, m, mask) for m in range(4)]


def _uneven_items(case, seed):
    """Sides log-uniform, template sides uniform, methods uniform; the sizes
    come from the case alone, the pixels from the seed."""
    shape = np.random.default_rng(3)
    g = _gen(seed)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    items = []
    for _ in range(case["n"]):
        W, H = (int(round(math.exp(v))) for v in shape.uniform(lo, hi, 2))
        w, h = (int(v) for v in shape.integers(case["tmin"], case["tmax"] + 1, 2))
        image = _uniform_u8((H, W), g)
        items.append((image, _crops(image, 1, w, h, g, 0, 4)[0].contiguous(), int(shape.integers(0, 4))))
    return items


def _scene(case, seed):
    """Value noise with 500 flat rectangles, and 48 x 48 crops of it."""
    g, side = _gen(seed), case["side"]
    image = _value_noise(side, side, g)
    shape = np.random.default_rng(seed)
    for _ in range(500):
        rw, rh = (int(v) for v in shape.integers(8, 256, 2))
        x, y = int(shape.integers(0, side - rw)), int(shape.integers(0, side - rh))
        image[y:y + rh, x:x + rw] = int(shape.integers(0, 256))
    return image, _crops(image, case["n"], 48, 48, g, 10, 6).contiguous()


def _training_inputs(case, seed):
    """Crops of value noise, a template of each and its position (downsampled)."""
    g, n, crop = _gen(seed), case["n"], case["crop"]
    crops = _crops(_value_noise(1024, 1024, g), n, crop, crop, g, 0, 0).contiguous()
    at = torch.randint(0, crop - 47, (2, n), generator=g, device="cuda")
    r = torch.arange(48, device="cuda")
    k = torch.arange(n, device="cuda")
    t = crops[k[:, None, None], (at[0][:, None] + r)[:, :, None], (at[1][:, None] + r)[:, None, :]].int()
    t = t + torch.randint(-6, 7, t.shape, generator=g, device="cuda", dtype=torch.int32)
    ds = crop // 4
    pos = (k * ds + (at[0] + 2) // 4 + 5) * ds + (at[1] + 2) // 4 + 5
    return crops, t.clamp(0, 255).to(torch.uint8).contiguous(), pos


def _score_map(case, seed):
    """A score map to suppress: CrossCorrelationNormalized of a 32 x 32 crop."""
    g = _gen(seed)
    image = _value_noise(case["W"] + 31, case["H"] + 31, g)
    return device.match_template_device(image, _crops(image, 1, 32, 32, g, 0, 6)[0].contiguous(), CCORR_NORM)


def _filter_inputs(case, seed):
    g = _gen(seed)
    W, H, ch = case["W"], case["H"], case["channels"]
    image = _value_noise(W, H, g)
    if ch > 1:
        image = torch.stack([image] * ch, 2) ^ _uniform_u8((H, W, ch), g) % 16
    taps = torch.rand((case["kh"], case["kw"]), generator=g, device="cuda") + 0.1
    kernel = taps / taps.sum() if case["float"] else (taps * 8).int() - 4
    return image.contiguous(), kernel.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("map", "host_map"):
        s["image"], s["template"], mask = _match_inputs(case, seed)
        s["mask"] = mask if case.get("mask") else None
        if kind == "host_map":
            s["image"], s["template"] = s["image"].cpu().numpy(), s["template"].cpu().numpy()
    elif kind in ("eight", "uneven"):
        items = _eight_items(case, seed) if kind == "eight" else _uneven_items(case, seed)
        s["batch"] = device.Batch(items, extremes=kind == "uneven")
        s["plan"] = device.BatchPlan(s["batch"])
    elif kind == "many":
        g = _gen(seed)
        s["image"] = _value_noise(case["W"], case["H"], g)
        s["templates"] = _crops(s["image"], case["n"], case["w"], case["h"], g, 0, 6).contiguous()
    elif kind == "propose":
        s["image"], s["templates"] = _scene(case, seed)
        s["net"] = learned.ProposalNet.trained()
    elif kind == "gradients":
        s["crops"], s["templates"], s["pos"] = _training_inputs(case, seed)
        s["net"] = learned.ProposalNet.trained()
    elif kind == "suppress":
        s["map"] = _score_map(case, seed)
        s["out"] = torch.empty_like(s["map"])
    elif kind == "integral":
        shape = (case["H"], case["W"]) if case["channels"] == 1 else (case["H"], case["W"], case["channels"])
        s["image"] = _uniform_u8(shape, _gen(seed))
        s["out"] = torch.empty((case["H"] + 1, case["W"] + 1) + shape[2:], device="cuda",
                               dtype=torch.int32 if case["bits"] == 32 else torch.int64)
    else:
        s["image"], s["kernel"] = _filter_inputs(case, seed)
        s["out"] = torch.empty(s["image"].shape, device="cuda",
                               dtype={U8: torch.uint8, I16: torch.int16, F32: torch.float32}[case["out"]])
    return s


# ---- one pass ---------------------------------------------------------------------

def _extremes(e):
    return [float(e.max_value), float(e.min_value), *e.max_value_location, *e.min_value_location]


def _call(name, *args):
    fn = getattr(_lib.lib(), name)
    fn.argtypes = [ctypes.c_void_p if a is None or isinstance(a, torch.Tensor) else ctypes.c_uint32
                   if isinstance(a, int) else type(a) for a in args]
    fn.restype = ctypes.c_int
    _lib.check(fn(*(a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args)))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "map":
        scores = device.match_template_device(state["image"], state["template"], case["method"], state["mask"],
                                              mask_is_binary=True)
        if not case["extremes"]:
            return scores
        return scores, _extremes(device.find_extremes_device(scores))
    if kind == "host_map":
        return tm.match_template(state["image"], state["template"], case["method"])
    if kind == "eight":
        return state["plan"].launch()
    if kind == "uneven":
        return state["plan"].launch(), state["batch"].extremes
    if kind == "many":
        scores, ex = device.match_templates_device(state["image"], state["templates"], case["method"],
                                                   extremes=True)
        return scores, np.array([_extremes(e) for e in ex])
    if kind == "propose":
        answers = state["net"].propose_and_match(state["image"], state["templates"])
        return {"value": np.array([a.value for a in answers]),
                "location": np.array([a.location for a in answers]),
                "margin": np.array([a.margin for a in answers], np.float32),
                "path": np.array([[a.path, a.uncertified] for a in answers])}
    if kind == "gradients":
        return state["net"].gradients(state["crops"], state["templates"], state["pos"])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    W, H = case["W"], case["H"]
    if kind == "suppress":
        _call("ipb_suppress_non_maximum_f32_device", state["map"], W, H, case["r"], state["out"], stream)
    elif kind == "integral":
        _call("ipb_integral_image_device", state["image"], W, H, case["channels"], int(case["squared"]),
              case["bits"], state["out"], stream)
    else:
        _call("ipb_filter_clamped_device", state["image"], W, H, case["channels"], state["kernel"],
              0 if case["float"] else 1, case["kw"], case["kh"], case["out"], state["out"], stream)
    return state["out"]


# ---- the work of a pass -------------------------------------------------------------

def _map_work(W, H, w, h, masked):
    pos = (W - w + 1) * (H - h + 1)
    return W * H + w * h * (2 if masked else 1) + 4 * pos, 2 * pos * w * h


def work(case):
    kind = case["kind"]
    if kind in ("map", "host_map"):
        b, f = _map_work(case["W"], case["H"], case["w"], case["h"], case.get("mask"))
        return {"bytes": b, "flops": f}
    if kind == "eight":
        b, f = _map_work(case["W"], case["H"], case["w"], case["h"], True)
        return {"bytes": 8 * b - 7 * case["W"] * case["H"], "flops": 8 * f}
    if kind == "uneven":
        shape = np.random.default_rng(3)
        total = [0, 0]
        for _ in range(case["n"]):
            W, H = (int(round(math.exp(v))) for v in shape.uniform(math.log(case["lo"]), math.log(case["hi"]), 2))
            w, h = (int(v) for v in shape.integers(case["tmin"], case["tmax"] + 1, 2))
            shape.integers(0, 4)
            b, f = _map_work(W, H, w, h, False)
            total[0] += b
            total[1] += f
        return {"bytes": total[0], "flops": total[1]}
    if kind == "many":
        pos = (case["W"] - case["w"] + 1) * (case["H"] - case["h"] + 1)
        tp = case["w"] * case["h"]
        return {"bytes": case["W"] * case["H"] + case["n"] * (tp + 4 * pos), "flops": 2 * pos * tp * case["n"]}
    if kind in ("propose", "gradients"):
        # the network's convolutions on the 4x-downsampled pixels and its heatmap
        n = case["n"]
        if kind == "propose":
            px = case["side"] ** 2 // 16 + 144 * n
            flops = px * 2 * 9 * 32 * (1 + 4 * 32) + 2 * 128 * n * px
            return {"bytes": case["side"] ** 2 + 48 * 48 * n, "flops": flops}
        px = n * (case["crop"] ** 2 // 16 + 144)
        flops = 3 * (px * 2 * 9 * 32 * (1 + 4 * 32) + 2 * 128 * n * px)
        return {"bytes": 16 * px + 8 * learned.N_PARAMS, "flops": flops}
    px = case["W"] * case["H"]
    if kind == "suppress":
        return {"bytes": 8 * px, "flops": 4 * px}
    if kind == "integral":
        ch = case["channels"]
        return {"bytes": px * ch + (case["W"] + 1) * (case["H"] + 1) * ch * case["bits"] // 8, "flops": 3 * px * ch}
    ch = case["channels"]
    return {"bytes": px * ch * (1 + {U8: 1, I16: 2, F32: 4}[case["out"]]), "flops": 2 * px * ch * case["kw"] * case["kh"]}


# ---- exact results --------------------------------------------------------------------

def _correlate(image, template):
    """Exact integer correlation (as float64) through an FFT in 64 bits."""
    H, W = image.shape
    h, w = template.shape
    s = (H, W)
    spec = torch.fft.rfft2(image.double(), s=s) * torch.fft.rfft2(template.double(), s=s).conj()
    return torch.fft.irfft2(spec, s=s)[:H - h + 1, :W - w + 1].round()


def _box(image, w, h):
    s = F.pad(image.double().cumsum(0).cumsum(1), (1, 0, 1, 0))
    return s[h:, w:] - s[:-h, w:] - s[h:, :-w] + s[:-h, :-w]


def _exact_scores(image, template, method, mask=None):
    h, w = template.shape
    t = template.double() if mask is None else template.double() * mask
    square = image.double().square()
    x = _correlate(image, t if mask is None else t * mask)
    y = _box(square, w, h) if mask is None else _correlate(square, mask.double().square())
    tss = t.square().sum()
    score = x if method in (CCORR, CCORR_NORM) else y + tss - 2 * x
    if method in (SSE, CCORR):
        return score
    norm = (y * tss).sqrt()
    return torch.where(norm > 0, score / norm.clamp(min=1e-300), score)


def _bf16(v):
    """v rounded to bf16, with the gradient of the identity: the network's
    weights and activations are bf16 values."""
    return v + (v.detach().bfloat16().double() - v.detach())


def _net(params, images):
    """The proposal network's features, summed in 64 bits."""
    a = (F.avg_pool2d(images.double()[:, None], 4) * 16 - 2048) / 1024
    for k, (weight, bias) in enumerate(params):
        a = F.conv2d(a, _bf16(weight), bias, padding=1)
        a = _bf16(a.relu() if k < 4 else a)
    return a


def _exact_gradients(case, seed):
    crops, templates, pos = _training_inputs(case, seed)
    flat = torch.from_numpy(np.load(learned.WEIGHTS)).cuda().double()
    params, off = [], 0
    for cin in NET_LAYERS:
        n = 32 * cin * 9
        params.append((flat[off:off + n].reshape(32, cin, 3, 3).requires_grad_(),
                       flat[off + n:off + n + 32].requires_grad_()))
        off += n + 32
    f = _net(params, crops)
    t = _net(params, templates)[:, :, 5:7, 5:7]
    z = F.conv2d(F.pad(f, (0, 1, 0, 1)), t) / 8   # (crops, templates, y, x)
    n, ds = case["n"], case["crop"] // 4
    y, x = (pos % (ds * ds)) // ds, pos % ds
    yy, xx = torch.arange(ds, device="cuda")[:, None], torch.arange(ds, device="cuda")[None]
    near = ((yy - y[:, None, None]).abs() <= 1) & ((xx - x[:, None, None]).abs() <= 1)
    own = z[pos // (ds * ds), torch.arange(n, device="cuda")]
    positive = own.masked_fill(~near, -math.inf).flatten(1).logsumexp(1)
    loss = (z.transpose(0, 1).flatten(1).logsumexp(1) - positive).mean()
    grads = torch.autograd.grad(loss, [p for pair in params for p in pair])
    return float(loss.detach()), torch.cat([v.flatten() for v in grads])


def _exact_suppress(case, seed):
    """The pixels that are the greatest of their window; the smaller (x, y) wins."""
    m, r = _score_map(case, seed), case["r"]
    H, W = m.shape
    keep = (F.max_pool2d(m[None, None], 2 * r + 1, 1, r)[0, 0] == m).nonzero()
    d = torch.arange(-r, r + 1, device="cuda")
    dy, dx = d.repeat_interleave(2 * r + 1), d.repeat(2 * r + 1)
    first = (dx < 0) | ((dx == 0) & (dy < 0))
    out = torch.zeros_like(m, dtype=torch.float64)
    for part in keep.split(1 << 16):
        y, x = part[:, :1] + dy[first], part[:, 1:] + dx[first]
        inside = (y >= 0) & (y < H) & (x >= 0) & (x < W)
        v = m[part[:, 0], part[:, 1]]
        beaten = (inside & (m[y.clamp(0, H - 1), x.clamp(0, W - 1)] == v[:, None])).any(1)
        part, v = part[~beaten], v[~beaten]
        out[part[:, 0], part[:, 1]] = v.double()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("map", "host_map"):
        image, template, mask = _match_inputs(case, seed)
        scores = _exact_scores(image, template, case["method"], mask if case.get("mask") else None)
        return (scores, None) if case.get("extremes") else scores
    if kind == "eight":
        return [_exact_scores(*item) for item in _eight_items(case, seed)]
    if kind == "uneven":
        return [_exact_scores(*item) for item in _uneven_items(case, seed)], None
    if kind == "many":
        s = prepare(case, seed)
        H, W = case["H"] - case["h"] + 1, case["W"] - case["w"] + 1
        out = torch.empty((H, W, case["n"]), dtype=torch.float64, device="cuda")
        for k in range(case["n"]):
            out[:, :, k] = _exact_scores(s["image"], s["templates"][k], case["method"])
        return out, None
    if kind == "propose":
        image, templates = _scene(case, seed)
        value = [float(_exact_scores(image, t, SSE).min()) for t in templates]
        return {"value": np.array(value), "location": None, "margin": None, "path": None}
    if kind == "gradients":
        return _exact_gradients(case, seed)
    if kind == "suppress":
        return _exact_suppress(case, seed)
    if kind == "filter" and case["out"] == F32:
        image, kernel = _filter_inputs(case, seed)
        planes = (image if image.dim() == 3 else image[..., None]).permute(2, 0, 1)[:, None].double()
        kh, kw = kernel.shape
        planes = F.pad(planes, (kw // 2, kw - 1 - kw // 2, kh // 2, kh - 1 - kh // 2), mode="replicate")
        out = F.conv2d(planes, kernel.double()[None, None])[:, 0].permute(1, 2, 0)
        return out.reshape(image.shape)
    return None
