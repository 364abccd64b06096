"""The work a user of this framework has it do, as timed cases.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` what a
program holds before the call, ``run(state)`` one pass through the public entry points, ``work(case)`` the
bytes and operations of one pass that no implementation can do without.

Kinds of case:

* ``encode`` / ``decode``: one texture on the device (``capi``: ``qt_bc*_encode_device`` /
  ``_decode_device``), as engines and asset pipelines with resident texels call it;
* ``dropin``: ``BC1Encoder(level).encode(RawTexture)`` and the decode of its result on host textures, the
  ``quicktex`` interface;
* ``batch``: many textures of mixed sizes, formats, levels and directions in one launch (``Batch.run``);
* ``mips``: a mip chain resized from its top level on the device, all levels encoded in one launch.

Outputs are bytes (blocks or texels), so no value has an exact counterpart: ``exact`` is ``None``.
"""

import math
import random

import numpy as np
import torch

import quicktex_b200 as qt
from quicktex_b200 import batch, capi, image_utils
from quicktex_b200.s3tc import bc1, interpolator

FMT = {"bc1": 1, "bc3": 3, "bc4": 4, "bc5": 5}
BLOCK_BYTES = {"bc1": 8, "bc3": 16, "bc4": 8, "bc5": 16}
MODES = {"four": capi.FOUR_COLOR, "three": capi.THREE_COLOR, "black": capi.THREE_COLOR_BLACK}
INTERPOLATORS = {"ideal": capi.IDEAL, "round": capi.IDEAL_ROUND, "nvidia": capi.NVIDIA, "amd": capi.AMD}


def _encode(fmt, w, h, level=5, mode="four", interp="ideal"):
    return {"kind": "encode", "fmt": fmt, "w": w, "h": h, "level": level, "mode": mode, "interp": interp}


def _decode(fmt, w, h, interp="ideal"):
    return {"kind": "decode", "fmt": fmt, "w": w, "h": h, "interp": interp}


def listed():
    return [
        # the smallest call: an icon at the default level, where launches and latency count
        dict(_encode("bc3", 64, 64), name="bc3-l5-64"),
        # the quicktex interface on a small host texture: encode at the default level, then decode
        {"name": "dropin-bc1-l5-256", "kind": "dropin", "w": 256, "h": 256, "level": 5, "mode": "four", "interp": "ideal"},
        # an ordinary host texture at the top quality level of the quicktex interface (offline builds)
        {"name": "dropin-bc1-l18-1024", "kind": "dropin", "w": 1024, "h": 1024, "level": 18, "mode": "four", "interp": "ideal"},
        # a small texture off the 4-texel grid at the top level, all colour modes tried, a GPU vendor's interpolation
        dict(_encode("bc1", 510, 334, 18, "black", "nvidia"), name="bc1-l18-black-510x334"),
        # large colour textures: the fastest level, the middle of the range, the top level
        dict(_encode("bc1", 4096, 4096, 0), name="bc1-l0-4096"),
        dict(_encode("bc1", 2048, 2048, 10, "three"), name="bc1-l10-three-2048"),
        dict(_encode("bc1", 4096, 4096, 18), name="bc1-l18-4096"),
        # a large tangent-space normal map
        dict(_encode("bc5", 8192, 8192), name="bc5-8192"),
        # a single-channel map whose sides are not multiples of 4 (scans, atlases, lookup tables)
        dict(_encode("bc4", 4095, 4097), name="bc4-4095x4097"),
        # decoding a ragged texture (asset conversion, thumbnails)
        dict(_decode("bc1", 2002, 3001), name="bc1-decode-2002x3001"),
        # a folder of mixed textures in one launch: sizes 4 to 2048, formats 4:3:2:1, levels 0/5/10/18, 30% decodes
        {"name": "batch-500", "kind": "batch", "count": 500, "largest": 2048, "mix": 1},
        # the mip chain of an RGBA texture, every level from the top one, then BC3
        {"name": "mips-bc3-l10-2048", "kind": "mips", "fmt": "bc3", "w": 2048, "h": 2048, "level": 10},
    ]


# candidate evaluations (one texel against one palette colour) of a block at a preset level, about
def _evaluations(level, mode):
    p = capi.params_for_level(level, MODES[mode])
    orderings4, orderings3 = (969, 153) if p.exhaustive else (p.orderings4, p.orderings3)
    passes = 2 if p.two_cf_passes else 1
    trials = (2 if p.two_ep_passes else 1) * (1 + (1.5 if p.two_ls_passes else 1)) + orderings4 * passes
    trials += min(p.search_rounds, 34)
    three = 0 if mode == "four" else 1 + (1.5 if p.two_ls_passes else 1) + orderings3 * passes
    # two of four colours are tried per texel in the Check2 mode, one in Faster, all in Full
    per = {0: 16, 1: 16, 2: 32, 3: 64}[p.error_mode]
    return trials * per + three * 48


_LARGEST = 4096 * 4096 // 16 * 13000.0  # evaluations of the largest listed encode


def _side(rng, lo, hi):
    s = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return s if rng.random() < 0.4 else max(lo, (s + 2) // 4 * 4)


def draw(rng):
    kind = rng.choice(["bc1", "bc1", "bc1", "bc3", "bc45", "bc45", "decode", "decode", "dropin", "dropin", "batch", "mips"])
    interp = rng.choice(list(INTERPOLATORS))
    if kind == "decode":
        return _decode(rng.choice(list(FMT)), _side(rng, 64, 8192), _side(rng, 64, 8192), interp)
    if kind == "bc45":
        return _encode(rng.choice(["bc4", "bc5"]), _side(rng, 64, 8192), _side(rng, 64, 8192))
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(20, 500), "largest": rng.choice([256, 512, 1024, 2048]), "mix": rng.randrange(1 << 20)}
    if kind == "mips":
        return {"kind": "mips", "fmt": rng.choice(["bc1", "bc3"]), "w": _side(rng, 64, 2048), "h": _side(rng, 64, 2048),
                "level": rng.choice([0, 5, 10])}
    level = rng.choice(list(range(20)) + [0, 5, 5, 10, 18, 18])
    mode = "four" if kind == "bc3" else rng.choice(list(MODES))
    top = min(4096.0, math.sqrt(16 * _LARGEST / _evaluations(level, mode)))
    if kind == "dropin":
        top = min(top, 2048.0)
    w, h = _side(rng, 16, top), _side(rng, 16, top)
    if kind == "dropin":
        return {"kind": "dropin", "w": w, "h": h, "level": level, "mode": mode, "interp": interp}
    return _encode(kind, w, h, level, mode, interp)


# ---- inputs -------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _texture(w, h, g, alpha=False):
    """RGBA8 texels: of the 4x4 blocks 40% are gradients with noise, 30% uniform random, 20% two colours
    along an edge, 10% one colour; alpha 255, or per block a cutout, a ramp or noise."""
    bw, bh = (w + 3) // 4, (h + 3) // 4
    rnd = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731
    pos = torch.arange(4, device="cuda", dtype=torch.float32) - 1.5
    img = torch.empty(bh * 4, bw * 4, 4, dtype=torch.uint8, device="cuda")
    rows = max(1, (1 << 19) // bw)  # block rows made at a time
    for r in range(0, bh, rows):
        n = min(rows, bh - r)
        kind = rnd(n, bw, 1, 1, 1)
        c0, c1 = (rnd(n, bw, 1, 1, 3) * 255 for _ in range(2))
        angle = rnd(n, bw, 1, 1, 1) * (2 * math.pi)
        along = (torch.cos(angle) * pos.view(1, 1, 1, 4, 1) + torch.sin(angle) * pos.view(1, 1, 4, 1, 1)) / 4.3 + 0.5
        t = along.clamp(0, 1)
        gradient = c0 + (c1 - c0) * t + (rnd(n, bw, 4, 4, 3) * 16 - 8)
        edge = torch.where(along > 0.3 + 0.4 * rnd(n, bw, 1, 1, 1), c0, c1).expand(n, bw, 4, 4, 3)
        rgb = torch.where(kind < 0.4, gradient, torch.where(kind < 0.7, rnd(n, bw, 4, 4, 3) * 255,
                                                            torch.where(kind < 0.9, edge, c0.expand(n, bw, 4, 4, 3))))
        if alpha:
            k = rnd(n, bw, 1, 1, 1)
            a = torch.where(k < 0.34, (along > 0.5) * 255.0, torch.where(k < 0.67, t * 255, rnd(n, bw, 4, 4, 1) * 255))
        else:
            a = torch.full((n, bw, 4, 4, 1), 255.0, device="cuda")
        block = torch.cat([rgb, a], -1).round().clamp(0, 255).to(torch.uint8)
        img[r * 4: (r + n) * 4] = block.permute(0, 2, 1, 3, 4).reshape(n * 4, bw * 4, 4)
    return img[:h, :w].contiguous()


def _normals(w, h, g):
    """RGBA8 texels of a tangent-space normal map: x and y of the normals of eight smooth bumps."""
    x = (torch.arange(w, device="cuda", dtype=torch.float32) / max(w, h)).view(1, w)
    y = (torch.arange(h, device="cuda", dtype=torch.float32) / max(w, h)).view(h, 1)
    dx = torch.zeros(h, w, device="cuda")
    dy = torch.zeros(h, w, device="cuda")
    for cx, cy, size, height in torch.rand(8, 4, device="cuda", generator=g).tolist():
        s = 0.05 + 0.2 * size
        bump = (height - 0.3) * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * s * s)) / (s * s)
        dx += bump * (x - cx) * 0.3
        dy += bump * (y - cy) * 0.3
    length = torch.sqrt(dx * dx + dy * dy + 1)
    img = torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")
    img[..., 0] = ((dx / length * 0.5 + 0.5) * 255).round().to(torch.uint8)
    img[..., 1] = ((dy / length * 0.5 + 0.5) * 255).round().to(torch.uint8)
    img[..., 3] = 255
    return img


def _source(fmt, w, h, g):
    return _normals(w, h, g) if fmt == "bc5" else _texture(w, h, g, alpha=fmt == "bc3")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _params(level, mode, interp):
    return capi.params_for_level(level, MODES[mode], INTERPOLATORS[interp])


def _encode_call(fmt, src, w, h, params, dst):
    a, b = src.data_ptr(), dst.data_ptr()
    if fmt == "bc1":
        capi.bc1_encode_device(a, w, h, params, b, _stream())
    elif fmt == "bc3":
        capi.bc3_encode_device(a, w, h, params, b, _stream())
    elif fmt == "bc4":
        capi.bc4_encode_device(a, w, h, 0, b, _stream())
    else:
        capi.bc5_encode_device(a, w, h, 0, 1, b, _stream())


def _decode_call(fmt, src, w, h, interp, dst):
    L, a, b, s = capi.lib(), src.data_ptr(), dst.data_ptr(), _stream()
    if fmt == "bc1":
        capi.bc1_decode_device(a, w, h, interp, True, b, s)
    elif fmt == "bc3":
        capi.check(L.qt_bc3_decode_device(a, w, h, interp, b, s))
    elif fmt == "bc4":
        capi.check(L.qt_bc4_decode_device(a, w, h, 0, b, s))
    else:
        capi.check(L.qt_bc5_decode_device(a, w, h, 0, 1, b, s))


def _blocks(fmt, w, h):
    return torch.zeros(capi.nblocks(w, h) * BLOCK_BYTES[fmt], dtype=torch.uint8, device="cuda")


def _encoded(fmt, w, h, g, mode="three"):
    """Blocks as an encoder leaves them: a decoder's input."""
    src, dst = _source(fmt, w, h, g), _blocks(fmt, w, h)
    _encode_call(fmt, src, w, h, _params(5, mode, "ideal"), dst)
    torch.cuda.synchronize()
    return dst


def _batch_shapes(case):
    """The textures of a batch: the same for every seed of the contents."""
    rng = random.Random(case["mix"])
    shapes = []
    for _ in range(case["count"]):
        w, h = (int(round(math.exp(rng.uniform(math.log(4), math.log(case["largest"]))))) for _ in range(2))
        if rng.random() < 0.75:
            w, h = ((v + 3) // 4 * 4 for v in (w, h))
        fmt = rng.choice(["bc1"] * 4 + ["bc3"] * 3 + ["bc4"] * 2 + ["bc5"])
        shapes.append((fmt, w, h, rng.choice([0, 5, 10, 18]), rng.choice(["four", "three", "black"]) if fmt == "bc1" else "four",
                       rng.random() < 0.3))
    return shapes


def _align(n):
    return (n + 255) // 256 * 256


def _items(jobs, src, dst):
    return batch.items_array(jobs, src, dst)


def _job(fmt, w, h, level, mode, decode):
    none = np.zeros(0, np.uint8)
    if decode:
        return batch.Job.decode(fmt, none, w, h, write_alpha=True, channel=0)
    return batch.Job.encode(fmt, none, w, h, level=level, color_mode=MODES[mode], channel=0)


def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    if kind == "encode":
        fmt, w, h = case["fmt"], case["w"], case["h"]
        state = {"src": _source(fmt, w, h, g), "dst": _blocks(fmt, w, h),
                 "params": _params(case["level"], case["mode"], case["interp"])}
    elif kind == "decode":
        fmt, w, h = case["fmt"], case["w"], case["h"]
        state = {"src": _encoded(fmt, w, h, g), "dst": torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda"),
                 "interp": INTERPOLATORS[case["interp"]]}
    elif kind == "dropin":
        w, h = case["w"], case["h"]
        kinds = {"ideal": interpolator.Interpolator, "round": interpolator.InterpolatorRound,
                 "nvidia": interpolator.InterpolatorNvidia, "amd": interpolator.InterpolatorAMD}
        modes = {"four": bc1.BC1Encoder.ColorMode.FourColor, "three": bc1.BC1Encoder.ColorMode.ThreeColor,
                 "black": bc1.BC1Encoder.ColorMode.ThreeColorBlack}
        itp = kinds[case["interp"]]()
        texels = _texture(w, h, g).cpu().numpy().tobytes()
        state = {"texture": qt.RawTexture.frombytes(texels, w, h), "encoder": bc1.BC1Encoder(case["level"], modes[case["mode"]], itp),
                 "decoder": bc1.BC1Decoder(True, itp)}
    elif kind == "batch":
        srcs, sizes, jobs = [], [], []
        for fmt, w, h, level, mode, decode in _batch_shapes(case):
            job = _job(fmt, w, h, level, mode, decode)
            srcs.append(_encoded(fmt, w, h, g) if decode else _source(fmt, w, h, g))
            sizes.append(_align(job.out_bytes))
            jobs.append(job)
        dst = torch.zeros(sum(sizes), dtype=torch.uint8, device="cuda")
        at = (np.cumsum([0] + sizes[:-1]) + dst.data_ptr()).tolist()
        state = {"srcs": srcs, "dst": dst, "items": _items(jobs, [s.data_ptr() for s in srcs], at), "queue": batch.Batch(torch.cuda.current_device())}
    else:
        fmt, w, h = case["fmt"], case["w"], case["h"]
        sizes = image_utils.mip_sizes((w, h))
        jobs = [_job(fmt, a, b, case["level"], "four", False) for a, b in sizes]
        texels, blocks = ([_align(n) for n in ns] for ns in ([a * b * 4 for a, b in sizes], [j.out_bytes for j in jobs]))
        lv = torch.zeros(sum(texels), dtype=torch.uint8, device="cuda")
        lv[: w * h * 4] = _texture(w, h, g, alpha=True).view(-1)
        dst = torch.zeros(sum(blocks), dtype=torch.uint8, device="cuda")
        level_at = (np.cumsum([0] + texels[:-1]) + lv.data_ptr()).tolist()
        at = (np.cumsum([0] + blocks[:-1]) + dst.data_ptr()).tolist()
        state = {"levels": lv, "dst": dst, "sizes": sizes, "level_at": level_at, "items": _items(jobs, level_at, at),
                 "queue": batch.Batch(torch.cuda.current_device())}
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "encode":
        _encode_call(case["fmt"], state["src"], case["w"], case["h"], state["params"], state["dst"])
        return state["dst"]
    if kind == "decode":
        _decode_call(case["fmt"], state["src"], case["w"], case["h"], state["interp"], state["dst"])
        return state["dst"]
    if kind == "dropin":
        encoded = state["encoder"].encode(state["texture"])
        decoded = state["decoder"].decode(encoded)
        return [np.frombuffer(memoryview(encoded), np.uint8), np.frombuffer(memoryview(decoded), np.uint8)]
    if kind == "mips":
        (w0, h0), at, s = state["sizes"][0], state["level_at"], _stream()
        for (w, h), dst in zip(state["sizes"][1:], at[1:]):
            image_utils.resize_device(at[0], w0, h0, dst, w, h, s)
        state["queue"].run(state["items"], s)
        return [state["levels"], state["dst"]]
    state["queue"].run(state["items"], _stream())
    return state["dst"]


def work(case):
    def texture(fmt, w, h, level, mode, decode):
        n = capi.nblocks(w, h)
        flops = 0.0
        if not decode and fmt in ("bc1", "bc3"):
            flops = n * _evaluations(level, mode) * 8.0  # a squared distance over three channels
        return w * h * 4 + n * BLOCK_BYTES[fmt], flops

    kind = case["kind"]
    if kind == "batch":
        parts = [texture(*s) for s in _batch_shapes(case)]
    elif kind == "mips":
        sizes = image_utils.mip_sizes((case["w"], case["h"]))
        parts = [texture(case["fmt"], w, h, case["level"], "four", False) for w, h in sizes]
        # the top level read once for the smaller ones, each of them written; a resize multiplies and adds per tap
        top = case["w"] * case["h"]
        parts.append((sum(w * h * 4 for w, h in sizes[1:]), 2.0 * 4 * top * 2 * (len(sizes) - 1)))
    elif kind == "dropin":
        parts = [texture("bc1", case["w"], case["h"], case["level"], case["mode"], d) for d in (False, True)]
    else:
        parts = [texture(case["fmt"], case["w"], case["h"], case.get("level", 5), case.get("mode", "four"), kind == "decode")]
    return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(f for _, f in parts))}


def exact(case, seed):
    return None
