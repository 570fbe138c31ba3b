"""The calls that users of this library make, as measurable cases.

Every case is one pass through the public entry points on images that are
already on the GPU (the library takes device pointers), with the context, the
destination images and, for batches, the plan that a user's program keeps.

The listed cases are the uses; draw() gives further ones of the same ranges:

  op         sizes (log-uniform)      channels  options
  gauss      160..3840 x 120..2160    1, 3, 4   k 3 5 7 9 binomial, k 3..21 generated,
                                                four borders, 0..64 pad bytes per row
  arbitrary  320..3840 x 240..2160    1, 3      odd k 11..63, REPLICATE
  sep        160..3840 x 120..2160    1, 3      u8, u16, s16; five borders
  pyramid    512..8192 x 512..8192    1, 3, 4   2..6 levels
  sobel      160..3840 x 120..2160    1, 3, 4   both derivatives of one image
  median     160..1920 x 120..1080    1, 3      u8 k 3..15, u16 and f32 k 3 5
  batch      16..512 images, 64..4096 x 64..2160, k 3 5 7 15, one plan
"""
import importlib
import math
import random

import numpy as np
import torch

kcv = importlib.import_module("yocto-mirrors_gitlab_kleidi_kleidicv_gb300")

BORDERS = {"constant": kcv.CONSTANT, "replicate": kcv.REPLICATE, "reflect": kcv.REFLECT, "wrap": kcv.WRAP,
           "reverse": kcv.REVERSE}
CONSTANT_VALUE = 17
# Element types as torch holds them (u16 images travel as int16 bits).
TORCH_TYPES = {"u8": torch.uint8, "u16": torch.int16, "s16": torch.int16, "f32": torch.float32}


def listed():
    return [
        # The smallest call: a preview or a detector's input tile, where latency is all.
        {"name": "gauss_preview", "op": "gauss", "w": 320, "h": 240, "c": 1, "k": 5, "sigma": 0.0,
         "border": "replicate", "pad": 0},
        # One luma frame of a 1080p camera, rows padded by 64 bytes: denoising before detection.
        {"name": "gauss_1080p_luma", "op": "gauss", "w": 1920, "h": 1080, "c": 1, "k": 5, "sigma": 0.0,
         "border": "replicate", "pad": 64},
        # An RGBA 4K frame with a chosen sigma: the headline call of the benchmark.
        {"name": "gauss_4k_rgba", "op": "gauss", "w": 3840, "h": 2160, "c": 4, "k": 7, "sigma": 1.5,
         "border": "reverse", "pad": 0},
        # An RGB crop of odd size, tightly packed (no row is aligned), with a wide fixed kernel.
        {"name": "gauss_rgb_crop", "op": "gauss", "w": 1917, "h": 1079, "c": 3, "k": 15, "sigma": 2.5,
         "border": "reflect", "pad": 0},
        # Background or illumination estimate: a wide blur of a 4K luma frame.
        {"name": "gauss_wide", "op": "arbitrary", "w": 3840, "h": 2160, "c": 1, "k": 31, "sigma": 5.0,
         "border": "replicate", "pad": 0},
        # User taps on an RGB HD frame, 8 bits, with saturation in reach.
        {"name": "sep_u8_rgb", "op": "sep", "type": "u8", "w": 1280, "h": 720, "c": 3,
         "kx": "0 1 0 1 0", "ky": "0 0 1 0 0", "border": "reflect", "pad": 0},
        # User taps on a 4K 16-bit sensor frame.
        {"name": "sep_u16_4k", "op": "sep", "type": "u16", "w": 3840, "h": 2160, "c": 1,
         "kx": "0 1 2 1 0", "ky": "1 0 3 0 1", "border": "reflect", "pad": 0},
        # A 5-tap derivative of a signed frame of odd width, periodic border.
        {"name": "sep_s16_odd", "op": "sep", "type": "s16", "w": 3841, "h": 2161, "c": 1,
         "kx": "-1 -2 0 2 1", "ky": "1 4 6 4 1", "border": "wrap", "pad": 0},
        # An image pyramid of a large scan, five levels.
        {"name": "pyramid_scan", "op": "pyramid", "w": 8192, "h": 8192, "c": 1, "levels": 5,
         "border": "reverse", "pad": 0},
        # Both derivatives of a 1080p frame: edge detection.
        {"name": "sobel_1080p", "op": "sobel", "w": 1920, "h": 1080, "c": 1, "pad": 0},
        # Salt-and-pepper removal on a 1080p frame.
        {"name": "median_1080p", "op": "median", "type": "u8", "w": 1920, "h": 1080, "c": 1, "k": 5,
         "border": "replicate", "pad": 0},
        # A data loader's augmentation batch: 512 images of mixed sizes, channels and
        # kernels, tightly packed, one plan launched as a graph.
        {"name": "batch_mixed", "op": "batch", "images": 512, "mix": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gauss", "gauss", "gauss", "arbitrary", "sep", "sep", "pyramid", "sobel", "median", "batch"])
    fixed = ["replicate", "reflect", "wrap", "reverse"]
    pad = rng.choice([0, 0, 64, rng.randint(1, 63)])
    if op == "batch":
        return {"op": op, "images": _log_int(rng, 16, 320), "mix": rng.randint(10, 10 ** 6)}
    if op == "pyramid":
        c = rng.choice([1, 3, 4])
        return {"op": op, "w": _log_int(rng, 512, 8192 // (1 if c == 1 else 2)),
                "h": _log_int(rng, 512, 8192 // (1 if c == 1 else 2)), "c": c,
                "levels": rng.randint(2, 6), "border": rng.choice(fixed), "pad": pad}
    if op == "median":
        t = rng.choice(["u8", "u8", "u16", "f32"])
        return {"op": op, "type": t, "w": _log_int(rng, 160, 1920), "h": _log_int(rng, 120, 1080),
                "c": rng.choice([1, 3]), "k": rng.choice([3, 5, 7, 9, 15] if t == "u8" else [3, 5]),
                "border": rng.choice(fixed), "pad": 4 * (pad // 4)}
    w, h = _log_int(rng, 160, 3840), _log_int(rng, 120, 2160)
    if op == "gauss":
        k = rng.choice([3, 5, 7, 9, 15, 21])
        sigma = 0.0 if k <= 9 and rng.random() < 0.5 else round(rng.uniform(0.5, 4.0), 2)
        return {"op": op, "w": w, "h": h, "c": rng.choice([1, 3, 4]), "k": k, "sigma": sigma,
                "border": rng.choice(fixed), "pad": pad}
    if op == "arbitrary":
        return {"op": op, "w": max(w, 320), "h": max(h, 240), "c": rng.choice([1, 3]),
                "k": rng.choice([k for k in range(11, 64, 2) if k not in (15, 21)]),
                "sigma": round(rng.uniform(2.0, 10.0), 2), "border": "replicate", "pad": pad}
    if op == "sobel":
        return {"op": op, "w": w, "h": h, "c": rng.choice([1, 3, 4]), "pad": 2 * (pad // 2)}
    t = rng.choice(["u8", "u16", "s16"])
    taps = [" ".join(str(rng.randint(-4, 4) if t == "s16" else rng.randint(0, 3)) for _ in range(5)) for _ in range(2)]
    return {"op": "sep", "type": t, "w": w, "h": h, "c": rng.choice([1, 1, 3]), "kx": taps[0], "ky": taps[1],
            "border": rng.choice(fixed + ["constant"]), "pad": 2 * (pad // 2)}


# --- images ------------------------------------------------------------------

def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _rows(h, row_elems, pad_bytes, dtype):
    """An h x row_elems image whose rows are pad_bytes further apart."""
    es = torch.empty((), dtype=dtype).element_size()
    full = torch.zeros((h, row_elems + pad_bytes // es), dtype=dtype, device=_device())
    return full[:, :row_elems]


def _image(gen, w, h, c, pad, type_="u8"):
    """A frame: shaded surface with edges and sensor noise on the left, texture on the right."""
    dev = _device()
    lo, hi = {"u8": (0, 255), "u16": (0, 65535), "s16": (-32768, 32767), "f32": (0, 255)}[type_]
    x = torch.arange(w, device=dev, dtype=torch.float32).view(1, w, 1)
    y = torch.arange(h, device=dev, dtype=torch.float32).view(h, 1, 1)
    phase = torch.rand(c, generator=gen, device=dev) * 6.0
    noise = torch.rand((h, w, c), generator=gen, device=dev)
    v = 0.5 + 0.24 * torch.sin(x / 17.0 + y / 29.0 + phase) + 0.3 * (noise - 0.5)
    v = torch.where((x // 97 + y // 61) % 4 == 0, v - 0.25, v)
    v = torch.where(x >= w // 2, noise, v).clamp_(0.0, 1.0) * (hi - lo) + lo
    img = _rows(h, w * c, pad, TORCH_TYPES[type_])
    if type_ == "f32":
        img.copy_(v.view(h, w * c))
    else:
        v = v.round_().to(torch.int32).view(h, w * c)
        img.copy_(torch.where(v > 32767, v - 65536, v) if type_ == "u16" else v)
    return img


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _batch_spec(case):
    """Sizes, channels, kernels and borders of a batch's images."""
    rng = random.Random(case["mix"])
    spec = []
    for _ in range(case["images"]):
        spec.append({"w": _log_int(rng, 64, 4096), "h": _log_int(rng, 64, 2160), "c": rng.choice([1, 3, 4]),
                     "k": rng.choice([3, 5, 7, 15]), "sigma": rng.uniform(0.5, 4.0),
                     "border": rng.choice(["replicate", "reflect", "wrap", "reverse"])})
    return spec


def _arena(case):
    """One buffer for a batch's destinations (images 256 bytes aligned, rows
    tightly packed), and its images."""
    spec, offsets, total = _batch_spec(case), [], 0
    for p in spec:
        offsets.append(total)
        total += (p["w"] * p["h"] * p["c"] + 255) // 256 * 256
    flat = torch.zeros(total, dtype=torch.uint8, device=_device())
    return flat, [flat[o:o + p["w"] * p["h"] * p["c"]].view(p["h"], p["w"] * p["c"]) for o, p in zip(offsets, spec)]


def _source(case, seed):
    gen = _generator(seed)
    if case["op"] == "batch":
        return [torch.randint(0, 256, (s["h"], s["w"] * s["c"]), dtype=torch.uint8, device=_device(), generator=gen)
                for s in _batch_spec(case)]
    return _image(gen, case["w"], case["h"], case["c"], case["pad"], case.get("type", "u8"))


def _levels(case):
    w, h, sizes = case["w"], case["h"], []
    for _ in range(case["levels"]):
        w, h = (w + 1) // 2, (h + 1) // 2
        sizes.append((w, h))
    return sizes


def _taps(text):
    return [int(t) for t in text.split()]


def prepare(case, seed):
    src = _source(case, seed)
    st = {"case": case, "src": src, "ctx": kcv.Context.for_torch(0)}
    op, c = case["op"], case.get("c")
    if op == "batch":
        st["dst"], images = _arena(case)
        st["plan"] = kcv.BatchPlan(
            [kcv.make_request(kcv.OP_GAUSSIAN_BLUR_U8, kcv.ptr(s), kcv.stride(s), kcv.ptr(d), kcv.stride(d), p["w"],
                              p["h"], p["c"], p["k"], p["k"], p["sigma"], p["sigma"],
                              border_type=BORDERS[p["border"]])
             for s, d, p in zip(src, images, _batch_spec(case))], st["ctx"])
    elif op == "pyramid":
        st["dst"] = [_rows(h, w * c, case["pad"], torch.uint8) for w, h in _levels(case)]
    elif op == "sobel":
        st["dst"] = [_rows(case["h"], case["w"] * c, case["pad"], torch.int16) for _ in range(2)]
    else:
        st["dst"] = _rows(case["h"], case["w"] * c, case["pad"], src.dtype)
    if op == "sep":
        st["kx"], st["ky"] = _taps(case["kx"]), _taps(case["ky"])
    return st


def _ok(err):
    if err != kcv.OK:
        raise RuntimeError(f"call failed: {kcv.ERROR_NAMES.get(err, err)}")


def run(state):
    case, src, dst, ctx = state["case"], state["src"], state["dst"], state["ctx"]
    op = case["op"]
    if op == "batch":
        _ok(state["plan"].launch(True))
        return dst
    w, h, c = case["w"], case["h"], case["c"]
    if op == "pyramid":
        _ok(kcv.build_pyramid_u8(kcv.ptr(src), kcv.stride(src), w, h, c, [kcv.ptr(d) for d in dst],
                                 [kcv.stride(d) for d in dst], BORDERS[case["border"]], ctx))
    elif op == "sobel":
        _ok(kcv.sobel_3x3_horizontal_s16_u8(kcv.ptr(src), kcv.stride(src), kcv.ptr(dst[0]), kcv.stride(dst[0]),
                                            w, h, c, ctx))
        _ok(kcv.sobel_3x3_vertical_s16_u8(kcv.ptr(src), kcv.stride(src), kcv.ptr(dst[1]), kcv.stride(dst[1]),
                                          w, h, c, ctx))
    elif op == "sep":
        constant = case["border"] == "constant"
        _ok(kcv.separable_filter_2d(case["type"], kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h,
                                    c, state["kx"], 5, state["ky"], 5, BORDERS[case["border"]], ctx,
                                    border_value=CONSTANT_VALUE if constant else None))
    elif op == "median":
        _ok(kcv.median_blur(case["type"], kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h, c,
                            case["k"], case["k"], BORDERS[case["border"]], ctx))
    else:
        _ok(kcv.gaussian_blur_u8(kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h, c, case["k"],
                                 case["k"], case["sigma"], case["sigma"], BORDERS[case["border"]], ctx))
    return dst


def work(case):
    op = case["op"]
    if op == "batch":
        n = [(s["w"] * s["h"] * s["c"], s["k"]) for s in _batch_spec(case)]
        return {"bytes": sum(2 * e for e, _ in n), "flops": sum(4 * k * e for e, k in n)}
    n = case["w"] * case["h"] * case["c"]
    if op == "pyramid":
        out = sum(w * h for w, h in _levels(case)) * case["c"]
        # The levels below the last are outputs and inputs of one pass: written once.
        return {"bytes": n + out, "flops": 20 * out}
    if op == "sobel":
        return {"bytes": 5 * n, "flops": 14 * n}
    if op == "median":
        es = {"u8": 1, "u16": 2, "f32": 4}[case["type"]]
        return {"bytes": 2 * es * n, "flops": 2 * case["k"] * n}
    if op == "sep":
        return {"bytes": (2 if case["type"] == "u8" else 4) * n, "flops": 20 * n}
    return {"bytes": 2 * n, "flops": 4 * case["k"] * n}


# --- the same in 64-bit integers ------------------------------------------------

def _border_index(n, r, border):
    i = torch.arange(-r, n + r, device=_device())
    if border == "replicate":
        return i.clamp(0, n - 1)
    if border == "wrap":
        return i % n
    if border == "constant":
        return torch.where((i < 0) | (i >= n), torch.full_like(i, n), i)
    fold = 0 if border == "reflect" else 1
    i = torch.where(i < 0, -i - 1 + fold, i)
    return torch.where(i >= n, 2 * n - i - 1 - fold, i)


def _bordered(img, r, border):
    """h x w x c image with a mapped border of r pixels."""
    if border == "constant":
        img = torch.nn.functional.pad(img, (0, 0, 0, 1, 0, 1), value=CONSTANT_VALUE)
        h, w = img.shape[0] - 1, img.shape[1] - 1
    else:
        h, w = img.shape[:2]
    return img[_border_index(h, r, border)][:, _border_index(w, r, border)]


def _vertical(img, taps):
    h = img.shape[0] - len(taps) + 1
    return sum(int(t) * img[i:i + h] for i, t in enumerate(taps) if t)


def _horizontal(img, taps):
    w = img.shape[1] - len(taps) + 1
    return sum(int(t) * img[:, i:i + w] for i, t in enumerate(taps) if t)


BINOMIAL = {3: [1, 2, 1], 5: [1, 4, 6, 4, 1], 7: [2, 7, 14, 18, 14, 7, 2], 9: [4, 13, 30, 51, 60, 51, 30, 13, 4]}


def _gaussian_taps(k, sigma):
    """Weights in 1/256 with the rounding error carried along; [256] stands for a copy."""
    f = np.float32
    mid = k // 2
    s = f(sigma) if sigma else f(k) * f(0.15) + f(0.35)
    coef = f(1.0) / -(f(2.0) * s * s)
    g = [f(math.exp(float(f((mid - i) ** 2) * coef))) for i in range(mid)]
    total = f(0.0)
    for v in g:
        total = f(total + v)
    scale = f(256.0) / (total * f(2.0) + f(1.0))
    half, carried = [], f(0.0)
    for v in g:
        want = f(v * scale - carried)
        got = f(math.floor(float(want) + 0.5))
        half.append(int(got))
        carried = f(got - want)
    centre = int(math.floor(float(f(scale - carried)) + 0.5))
    return [256] if centre == 256 else half + [centre] + half[::-1]


def _gaussian(img, k, sigma, border):
    if k <= 9 and sigma == 0.0:
        taps = BINOMIAL[k]
        shift = 2 * int(round(math.log2(sum(taps))))
        v = _horizontal(_vertical(_bordered(img, k // 2, border), taps), taps)
        return (v + (1 << (shift - 1))) >> shift
    taps = _gaussian_taps(k, sigma)
    if taps == [256]:
        return img
    if sum(taps) > 256 and k not in (3, 5, 7, 9, 15, 21):
        return None  # wraps or saturates by position
    v = ((_vertical(_bordered(img, k // 2, border), taps) + 128) >> 8) & 255
    return ((_horizontal(v, taps) + 128) >> 8) & 255


def exact(case, seed):
    src = _source(case, seed)
    op = case["op"]
    if op == "batch":
        flat, images = _arena(case)
        for s, d, p in zip(src, images, _batch_spec(case)):
            d.copy_(_gaussian(s.view(p["h"], p["w"], p["c"]).long(), p["k"], p["sigma"], p["border"])
                    .reshape(p["h"], -1))
        return flat
    w, h, c = case["w"], case["h"], case["c"]
    if op == "median":
        k, n = case["k"], case["k"] ** 2
        wide = src.float() if case["type"] == "f32" else src.int()
        if case["type"] == "u16":
            wide = wide & 0xFFFF
        img = _bordered(wide.view(h, w, c), k // 2, case["border"])
        out, step = [], max(1, (1 << 26) // (w * c * n))
        for y in range(0, h, step):
            m = min(step, h - y)
            win = torch.stack([img[y + a:y + a + m, b:b + w] for a in range(k) for b in range(k)])
            out.append(win.sort(dim=0).values[n // 2])
        return torch.cat(out).to(src.dtype).reshape(h, -1)
    img = src.reshape(h, w, c).long()
    if op == "pyramid":
        out = []
        for _ in range(case["levels"]):
            v = _horizontal(_vertical(_bordered(img, 2, case["border"]), BINOMIAL[5]), BINOMIAL[5])
            img = ((v + 128) >> 8)[::2, ::2]
            out.append(img.to(torch.uint8).reshape(img.shape[0], -1))
        return out
    if op == "sobel":
        b = _bordered(img, 1, "replicate")
        return [_horizontal(_vertical(b, [1, 2, 1]), [-1, 0, 1]).to(torch.int16).reshape(h, -1),
                _horizontal(_vertical(b, [-1, 0, 1]), [1, 2, 1]).to(torch.int16).reshape(h, -1)]
    if op == "sep":
        hi = {"u8": 255, "u16": 65535, "s16": 32767}[case["type"]]
        if case["type"] == "u16":
            img = img & 0xFFFF
        v = _vertical(_bordered(img, 2, case["border"]), _taps(case["ky"]))
        if isinstance(v, int):
            v = torch.zeros_like(_bordered(img, 2, case["border"])[4:])
        if case["type"] != "s16":
            v = v.clamp(max=hi)
        o = _horizontal(v, _taps(case["kx"]))
        if isinstance(o, int):
            o = torch.zeros_like(img)
        o = o.clamp(-hi - 1 if case["type"] == "s16" else 0, hi)
        if case["type"] == "u16":
            o = torch.where(o > 32767, o - 65536, o)
        return o.to(src.dtype).reshape(h, -1)
    out = _gaussian(img, case["k"], case["sigma"], case["border"])
    return None if out is None or (op == "arbitrary" and c > 1) else out.to(torch.uint8).reshape(h, -1)
