"""The work that a user of the encoder has it do, as timed cases.

Kinds of case, each one pass through a public call of ``icbc_gb300``:

* ``image``  -- one RGBA8 image on the GPU, encoded by ``compress_image``
* ``blocks`` -- float blocks in the ``icbc::compress_bc1`` layout, by ``compress_blocks``
* ``batch``  -- many images of mixed size, level and decoder in a planned ``Batch``
* ``decode`` -- blocks decoded and measured against their texels
  (``decode_blocks`` and ``evaluate_errors``), a quality check's inner loop
* ``host``   -- an image in pinned host memory through ``compress_image_host``

Images are made on the GPU from the seed: bilinear gradients, four octaves of
value noise and hard-edged rectangles, with 5% single-colour and 5% near-black
blocks (``photo``), or the independent mixture of noise, dither, flat, dark
and gradient blocks with a quarter of the texels transparent (``mixture``).
"""
import math
import random

import torch

import icbc_gb300 as ig
from icbc_gb300 import synth

LUMA = (0.299, 0.587, 0.114)
FLAT = (1.0, 1.0, 1.0)


def _image(name, width, height, level, weights="alpha", luma=True, decoder=0, content="photo"):
    return {"name": name, "kind": "image", "width": width, "height": height, "level": level, "weights": weights,
            "luma": luma, "decoder": decoder, "content": content}


def listed():
    return [
        # An icon or one tile of an atlas, encoded when it changes: the smallest call, at the default quality.
        _image("tile_64_default", 64, 64, 8, "uniform", False),
        # One ordinary texture at the default quality, weights and colour weights left alone.
        _image("texture_512_default", 512, 512, 8, "uniform", False),
        # A picture whose sides are no multiple of four, at a middle quality, AMD's decoder.
        _image("odd_1021x763_level5", 1021, 763, 5, "alpha", False, decoder=2),
        # A large image at the fast setting: previews, textures made at run time.
        _image("large_4096_fast", 4096, 4096, 1),
        # The same at a middle quality, as a bulk conversion chooses it.
        _image("large_4096_level6", 4096, 4096, 6),
        # The default quality on a large image with transparency: the usual asset build.
        _image("large_4096_default", 4096, 4096, 8),
        # The final asset build: the best quality, with endpoint refinement.
        _image("large_4096_max", 4096, 4096, 9),
        # An importance map weighs the texels (float weights of the caller's own), NVIDIA's decoder.
        _image("plane_1000x600_default", 1000, 600, 8, "plane", True, decoder=1),
        # A caller of compress_bc1 with its own blocks of floats and weights, at the best quality.
        {"name": "blocks_40000_max", "kind": "blocks", "count": 40000, "level": 9, "weighted": True, "luma": True,
         "decoder": 0},
        # A build's images together: every size from 64 to 2048, every level, three decoders.
        {"name": "batch_300_mixed", "kind": "batch", "images": 300, "side_max": 2048, "mix": 1},
        # Checking an encoded image: decode the blocks and measure each against its texels.
        {"name": "decode_check_4096", "kind": "decode", "count": 1048576, "decoder": 0},
        # An image that lies in host memory, blocks wanted there: the whole call with its copies.
        {"name": "host_2048_default", "kind": "host", "width": 2048, "height": 2048, "level": 8, "weights": "alpha",
         "luma": True, "decoder": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image"] * 6 + ["blocks", "batch", "decode", "host"])
    decoder, luma = rng.randrange(4), rng.random() < 0.5
    weights = rng.choice(["uniform", "alpha", "alpha", "plane"])
    width, height = _log_int(rng, 64, 4096), _log_int(rng, 64, 4096)
    if rng.random() < 0.5:  # half of the sides whole blocks, as most textures have them
        width, height = max(64, width & ~3), max(64, height & ~3)
    level = rng.choice([0, 1, 2, 3, 4, 5, 6, 7, 8, 8, 8, 9, 9])
    if kind == "image":
        case = _image("", width, height, level, weights, luma, decoder, rng.choice(["photo", "photo", "mixture"]))
        del case["name"]
        return case
    if kind == "blocks":
        return {"kind": "blocks", "count": _log_int(rng, 256, 200000), "level": level, "weighted": rng.random() < 0.7,
                "luma": luma, "decoder": decoder}
    if kind == "batch":
        return {"kind": "batch", "images": _log_int(rng, 20, 300), "side_max": _log_int(rng, 256, 2048),
                "mix": rng.randrange(1 << 20)}
    if kind == "decode":
        return {"kind": "decode", "count": _log_int(rng, 256, 1 << 20), "decoder": decoder}
    return {"kind": "host", "width": min(width, 2048), "height": min(height, 2048), "level": level,
            "weights": weights if weights != "plane" else "alpha", "luma": luma, "decoder": decoder}


# ------------------------------------------------------------------ inputs --

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _value_noise(g, w, h, octaves=4):
    """Octaves of value noise in [0, 1) (the finest cells about two pixels), smoothstep between the lattice points."""
    side = max(w, h)
    base = max(2, side // (2 << octaves))
    out, total = torch.zeros((h, w), device="cuda"), 0.0
    for k in range(octaves):
        cells, amp = base << k, 1.0 / (1 << k)
        lattice = torch.rand((cells + 1, cells + 1), generator=g, device="cuda")

        def places(n):
            f = (torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * (cells / side)
            i = f.long().clamp_(max=cells - 1)
            t = f - i
            return i, t * t * (3 - 2 * t)

        (iy, ty), (ix, tx) = places(h), places(w)
        rows = lattice[:, ix] + (lattice[:, ix + 1] - lattice[:, ix]) * tx
        out += amp * (rows[iy] + (rows[iy + 1] - rows[iy]) * ty[:, None])
        total += amp
    return out / total


def _photo(g, w, h):
    """(h, w, 4) uint8: gradients + value noise + 20 rectangles, 5% flat and 5% near-black blocks, alpha a noise field."""
    img = torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")
    v = torch.linspace(0, 1, h, device="cuda")[:, None]
    u = torch.linspace(0, 1, w, device="cuda")[None, :]
    corners = torch.rand((3, 4), generator=g, device="cuda")
    for c in range(3):
        c00, c10, c01, c11 = corners[c]
        val = (c00 * (1 - u) + c10 * u) * (1 - v) + (c01 * (1 - u) + c11 * u) * v
        val = val + 0.3 * (_value_noise(g, w, h) - 0.5)
        img[:, :, c] = (val * 255 + 0.5).floor().clamp(0, 255).to(torch.uint8)
    for x, y, rw, rh, r, gr, b in torch.rand((20, 7), generator=g, device="cuda").tolist():
        x0, y0 = int(x * w), int(y * h)
        colour = torch.tensor([int(256 * r), int(256 * gr), int(256 * b)], dtype=torch.uint8, device="cuda")
        img[y0:y0 + 1 + int(rh * h / 4), x0:x0 + 1 + int(rw * w / 4), :3] = colour
    bw, bh = (w + 3) // 4, (h + 3) // 4
    spread = lambda t: t.repeat_interleave(4, 0).repeat_interleave(4, 1)[:h, :w]  # noqa: E731
    kind = spread(torch.rand((bh, bw), generator=g, device="cuda"))[:, :, None]
    flat = spread(torch.randint(0, 256, (bh, bw, 3), generator=g, device="cuda", dtype=torch.uint8))
    dark = torch.randint(0, 13, (h, w, 3), generator=g, device="cuda", dtype=torch.uint8)
    img[:, :, :3] = torch.where(kind < 0.05, flat, torch.where(kind < 0.10, dark, img[:, :, :3]))
    img[:, :, 3] = (_value_noise(g, w, h) * 255 + 0.5).floor().to(torch.uint8)
    return img


def _content(case, seed):
    w, h = case["width"], case["height"]
    if case.get("content") == "mixture":
        img = synth.hard_mixture_torch((w + 3) & ~3, (h + 3) & ~3, int(seed) * 7919 + 17)
        return img[:h, :w].contiguous()
    return _photo(_generator(seed), w, h)


def _encode_options(case):
    mode = {"uniform": ig.WEIGHTS_UNIFORM, "alpha": ig.WEIGHTS_ALPHA, "plane": ig.WEIGHTS_PLANE}[case["weights"]]
    return {"level": case["level"], "decoder": case["decoder"], "color_weights": LUMA if case["luma"] else FLAT,
            "weight_mode": mode}


def _simple_blocks(texels):
    """BC1 blocks of (n, 16, 4) texels by a plain range fit (extremes as endpoints), so that decoding reads blocks as
    an encoder makes them: most in the four-colour order, flat ones in the three-colour one."""
    rgb = texels[:, :, :3].to(torch.int32)
    hi, lo = rgb.amax(1), rgb.amin(1)
    pack = lambda c: ((c[:, 0] >> 3) << 11) | ((c[:, 1] >> 2) << 5) | (c[:, 2] >> 3)  # noqa: E731
    span = (hi - lo).sum(1).clamp(min=1)
    t = ((rgb - lo[:, None]).sum(2) * 3 + span[:, None] // 2) // span[:, None]  # 0 (low) .. 3 (high)
    code = torch.tensor([1, 3, 2, 0], dtype=torch.int32, device=texels.device)[t.long()]
    out = torch.empty((len(texels), 8), dtype=torch.uint8, device=texels.device)
    for k, c in ((0, pack(hi)), (2, pack(lo))):
        out[:, k], out[:, k + 1] = (c & 255).to(torch.uint8), (c >> 8).to(torch.uint8)
    shift = torch.arange(4, device=texels.device, dtype=torch.int32) * 2
    out[:, 4:] = (code.view(-1, 4, 4) << shift).sum(2).to(torch.uint8)
    return out


def _decode_inputs(case, seed):
    n = case["count"]
    bw = max(1, int(math.sqrt(n)))
    bh = -(-n // bw)
    img = _photo(_generator(seed), 4 * bw, 4 * bh)
    texels = img.view(bh, 4, bw, 4, 4).permute(0, 2, 1, 3, 4).reshape(-1, 16, 4)[:n].contiguous()
    return texels, _simple_blocks(texels)


def prepare(case, seed):
    ig.init(ig.Decoder_D3D10)
    kind = case["kind"]
    if kind == "image":
        options = _encode_options(case)
        if case["weights"] == "plane":
            options["weight_plane"] = _value_noise(_generator(seed + 1), case["width"], case["height"])
        return {"kind": kind, "rgba": _content(case, seed), "options": options}
    if kind == "host":
        rgba = _content(case, seed).cpu().pin_memory()
        blocks = ig.blocks_of(case["width"], case["height"])
        return {"kind": kind, "rgba": rgba.numpy(), "keep": rgba, "options": _encode_options(case),
                "out": torch.zeros((blocks, 8), dtype=torch.uint8).pin_memory().numpy()}
    if kind == "blocks":
        side = 4 * int(math.ceil(math.sqrt(case["count"])))
        img = synth.hard_mixture_torch(side, side, int(seed) * 7919 + 17)
        tex = img.view(side // 4, 4, side // 4, 4, 4).permute(0, 2, 1, 3, 4).reshape(-1, 16, 4)[:case["count"]]
        colours = tex.float() / 255.0
        weights = colours[:, :, 3].contiguous() if case["weighted"] else None
        return {"kind": kind, "colours": colours.contiguous(), "weights": weights, "level": case["level"],
                "decoder": case["decoder"], "luma": case["luma"]}
    if kind == "batch":
        rng = random.Random(case["mix"])
        photo = _photo(_generator(seed), 4096, 4096)
        sizes, images, options = [], [], []
        for _ in range(case["images"]):
            w, h = _log_int(rng, 64, case["side_max"]), _log_int(rng, 64, case["side_max"])
            if rng.random() >= 0.1:
                w, h = w & ~3, h & ~3
            x, y = rng.randrange(4096 - w + 1), rng.randrange(4096 - h + 1)
            images.append(photo[y:y + h, x:x + w].contiguous())
            sizes.append(ig.blocks_of(w, h))
            options.append((rng.randrange(10), rng.randrange(3)))
        out = torch.zeros((sum(sizes), 8), dtype=torch.uint8, device="cuda")
        descs, at = [], 0
        for img, n, (level, decoder) in zip(images, sizes, options):
            descs.append(ig.image_desc(img, level, out[at:at + n], decoder=decoder, color_weights=FLAT,
                                       weight_mode=ig.WEIGHTS_UNIFORM))
            at += n
        torch.cuda.synchronize()
        return {"kind": kind, "batch": ig.Batch(descs, keepalive=(images, out)), "out": out}
    texels, blocks = _decode_inputs(case, seed)
    return {"kind": kind, "texels": texels.view(-1, 64), "blocks": blocks, "decoder": case["decoder"]}


# -------------------------------------------------------------------- runs --

def run(state):
    kind = state["kind"]
    if kind == "image":
        return ig.compress_image(state["rgba"], **state["options"])
    if kind == "host":
        return ig.compress_image_host(state["rgba"], out=state["out"], **state["options"])
    if kind == "blocks":
        blocks, errors = ig.compress_blocks(state["colours"], state["weights"], state["level"],
                                            decoder=state["decoder"],
                                            color_weights=LUMA if state["luma"] else FLAT)
        return {"blocks": blocks, "errors": errors}
    if kind == "batch":
        state["batch"].launch()
        return state["out"]
    return {"rgba": ig.decode_blocks(state["blocks"], state["decoder"]),
            "errors": ig.evaluate_errors(state["texels"], state["blocks"], state["decoder"])}


def _blocks(case):
    if "count" in case:
        return case["count"]
    if case["kind"] == "batch":
        rng, n = random.Random(case["mix"]), 0
        for _ in range(case["images"]):
            w, h = _log_int(rng, 64, case["side_max"]), _log_int(rng, 64, case["side_max"])
            if rng.random() >= 0.1:
                w, h = w & ~3, h & ~3
            rng.randrange(4096 - w + 1), rng.randrange(4096 - h + 1), rng.randrange(10), rng.randrange(3)
            n += ((w + 3) // 4) * ((h + 3) // 4)
        return n
    return ((case["width"] + 3) // 4) * ((case["height"] + 3) // 4)


def work(case):
    """Texels read once, blocks written once.  Operations: for an encoded block the nearest of four palette entries
    and its error for 16 texels (what every level ends with); for a decoded one its palette and 16 squared differences.
    A search costs more, but how much of it a level needs is the encoder's own affair."""
    n = _blocks(case)
    if case["kind"] == "decode":
        return {"bytes": n * (8 + 64 + 8 + 64 + 4), "flops": n * 16 * 8}
    texel = 4
    if case["kind"] == "blocks":
        texel = 20 if case["weighted"] else 16
    elif case.get("weights") == "plane":
        texel = 8
    extra = 4 if case["kind"] == "blocks" else 0
    return {"bytes": n * (16 * texel + 8 + extra), "flops": n * 16 * 4 * 8}


def exact(case, seed):
    """The squared errors of a decoded block in 64 bits.  An encoder's blocks are whole numbers, and its errors belong
    to the blocks it chose."""
    if case["kind"] != "decode":
        return None
    texels, blocks = _decode_inputs(case, seed)
    b = blocks.to(torch.int64)
    ends = [b[:, 0] | (b[:, 1] << 8), b[:, 2] | (b[:, 3] << 8)]
    raw = [torch.stack([c >> 11, (c >> 5) & 63, c & 31], 1) for c in ends]
    p0, p1 = (torch.stack([(c[:, 0] << 3) | (c[:, 0] >> 2), (c[:, 1] << 2) | (c[:, 1] >> 4),
                           (c[:, 2] << 3) | (c[:, 2] >> 2)], 1) for c in raw)
    if case["decoder"] == 0:
        four, three = ((2 * p0 + p1) // 3, (2 * p1 + p0) // 3), (p0 + p1) // 2
    elif case["decoder"] == 2:
        four, three = ((43 * p0 + 21 * p1 + 32) >> 6, (43 * p1 + 21 * p0 + 32) >> 6), (p0 + p1 + 1) // 2
    elif case["decoder"] == 3:
        four, three = ((171 * p0 + 85 * p1 + 128) >> 8, (171 * p1 + 85 * p0 + 128) >> 8), (p0 + p1 + 1) // 2
    else:
        d = p1[:, 1] - p0[:, 1]
        quarter = torch.div(d, 4, rounding_mode="trunc")

        def nv(first, second, green):
            rb = ((2 * first + second) * 22) // 8
            return torch.stack([rb[:, 0], green // 256, rb[:, 2]], 1) & 255

        four = (nv(raw[0], raw[1], 256 * p0[:, 1] + quarter + 128 + 80 * d),
                nv(raw[1], raw[0], 256 * p1[:, 1] - quarter + 128 - 80 * d))
        half = ((raw[0] + raw[1]) * 33) // 8
        three = torch.stack([half[:, 0], (256 * p0[:, 1] + quarter + 128 + 128 * d) // 256, half[:, 2]], 1) & 255
    is4 = (ends[0] > ends[1])[:, None]
    palette = torch.stack([p0, p1, torch.where(is4, four[0], three), torch.where(is4, four[1], 0 * p0)], 1)
    index = ((b[:, 4:, None] >> (2 * torch.arange(4, device=b.device))) & 3).view(-1, 16)
    chosen = torch.gather(palette, 1, index[:, :, None].expand(-1, -1, 3))
    diff = (chosen - texels[:, :, :3].to(torch.int64)).double()
    return {"rgba": None, "errors": diff.square().sum((1, 2))}
