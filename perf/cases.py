"""Performance cases: the calls a user of texpresso_gb300 makes, over the
sizes, formats, algorithms and contents they make them with.

Every case goes through the public Python entry points: the host-buffer calls
(``Format.compress``, ``Format.compress_block_masked``), the stream-ordered
device calls (``compress_device``, ``decompress_device``), the mip producer
with the batched plan (``mip_batch_device``, ``Batch``) and the serving loop
(``Server``).  Outputs are the bytes those calls write (compressed blocks,
pixels, mip levels), so there is no rounding to compare: ``exact`` has no
value to give and bytes have to be equal.

Contents:
  ramp    per 4x4 block a noisy two-colour ramp, 10 % flat blocks, an alpha
          ramp per block (the repository's synthetic texture): nearly every
          block has 16 distinct colours
  opaque  the same with alpha 255
  photo   smooth multi-octave colour fields with one step of dither, opaque:
          repeated colours in a block are common, as in photographs
  cutout  photo with a hard-edged alpha mask (foliage, decals, UI): blocks
          that are partly or fully transparent
  noise   smooth one- or two-channel fields with +-3 dither (height and
          normal maps)
"""
import numpy as np
import torch

import texpresso_gb300 as tx
from texpresso_gb300 import workloads

_ALG = {"range": 0, "cluster": 1, "iterative": 2}
_FMT = {"bc1": 0, "bc2": 1, "bc3": 2, "bc4": 3, "bc5": 4}


def listed():
    return [
        # one 4x4 block from host memory (the reference's compress_block_masked:
        # editors and importers that visit blocks one at a time): pure latency
        {"name": "block_bc3_cluster", "kind": "block", "fmt": "bc3", "alg": "cluster", "content": "ramp",
         "mask": 0xFFFF},
        # an icon or a small decal already on the GPU: a launch that does not fill the chip
        {"name": "icon_bc1_cluster_256", "kind": "device", "fmt": "bc1", "alg": "cluster", "content": "opaque",
         "width": 256, "height": 256, "channels": 4, "aw": False},
        # a material texture with the default parameters, the repository's headline workload
        {"name": "tex_bc3_cluster_2048", "kind": "device", "fmt": "bc3", "alg": "cluster", "content": "ramp",
         "width": 2048, "height": 2048, "channels": 4, "aw": False},
        # a foliage atlas of odd size, colours weighted by alpha; rows are not 16-byte aligned
        {"name": "atlas_bc3_cluster_aw_1023x769", "kind": "device", "fmt": "bc3", "alg": "cluster",
         "content": "cutout", "width": 1023, "height": 769, "channels": 4, "aw": True},
        # an offline, best-quality export of an opaque texture
        {"name": "tex_bc1_iterative_2048", "kind": "device", "fmt": "bc1", "alg": "iterative", "content": "opaque",
         "width": 2048, "height": 2048, "channels": 4, "aw": False},
        # run-time compression of a rendered texture: the fast fit
        {"name": "tex_bc3_range_2048", "kind": "device", "fmt": "bc3", "alg": "range", "content": "ramp",
         "width": 2048, "height": 2048, "channels": 4, "aw": False},
        # a terrain height map, native single-channel input
        {"name": "height_bc4_r8_4096", "kind": "device", "fmt": "bc4", "alg": "cluster", "content": "noise",
         "width": 4096, "height": 4096, "channels": 1, "aw": False},
        # a normal map of ragged size stored as RGBA8, as the reference reads it
        {"name": "normal_bc5_rgba_2047x1025", "kind": "device", "fmt": "bc5", "alg": "cluster", "content": "noise",
         "width": 2047, "height": 1025, "channels": 4, "aw": False},
        # reading a compressed texture back to RGBA8
        {"name": "decode_bc3_2048", "kind": "decode", "fmt": "bc3", "alg": "range", "content": "ramp",
         "width": 2048, "height": 2048},
        # the reference's own call: a photograph in host memory, blocks back in host memory
        {"name": "host_bc1_cluster_1024", "kind": "host", "fmt": "bc1", "alg": "cluster", "content": "photo",
         "width": 1024, "height": 1024, "aw": False},
        # a level's worth of textures of mixed sizes, formats and algorithms: mip chains, then one batch launch
        {"name": "batch_64_textures_mips", "kind": "batch", "textures": 64, "min_side": 4, "max_side": 2048,
         "spread": 7},
        # asset-server traffic: requests from host memory with mip chains, best-quality fit
        {"name": "serve_24_requests", "kind": "serve", "requests": 24, "min_side": 64, "max_side": 1024,
         "spread": 3},
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))))


def draw(rng):
    kind = rng.choice(["device"] * 8 + ["decode", "decode", "host", "host", "batch", "serve", "block"])
    if kind == "block":
        return {"kind": "block", "fmt": rng.choice(["bc1", "bc2", "bc3", "bc4", "bc5"]),
                "alg": rng.choice(["range", "cluster", "iterative"]),
                "content": rng.choice(["ramp", "opaque", "photo", "cutout"]), "mask": rng.choice([0xFFFF, rng.randrange(1, 0xFFFF)])}
    if kind == "batch":
        return {"kind": "batch", "textures": _log_int(rng, 4, 64), "min_side": 4,
                "max_side": rng.choice([128, 512, 1024]), "spread": rng.randrange(1000)}
    if kind == "serve":
        return {"kind": "serve", "requests": _log_int(rng, 2, 24), "min_side": 64,
                "max_side": rng.choice([128, 512, 1024]), "spread": rng.randrange(1000)}
    w, h = _log_int(rng, 4, 2048), _log_int(rng, 4, 2048)
    if rng.random() < 0.5:  # whole blocks and aligned rows half of the time, any size otherwise
        w, h = (w + 3) // 4 * 4, (h + 3) // 4 * 4
    if kind == "decode":
        return {"kind": "decode", "fmt": rng.choice(["bc1", "bc2", "bc3", "bc4", "bc5"]), "alg": "range",
                "content": rng.choice(["ramp", "opaque", "photo", "cutout"]), "width": w, "height": h}
    if kind == "device" and rng.random() < 0.3:
        fmt = rng.choice(["bc4", "bc5"])
        return {"kind": "device", "fmt": fmt, "alg": "cluster", "content": "noise", "width": w, "height": h,
                "channels": rng.choice([4, 1 if fmt == "bc4" else 2]), "aw": False}
    case = {"kind": kind, "fmt": rng.choice(["bc1", "bc1", "bc2", "bc3", "bc3"]),
            "alg": rng.choice(["range", "cluster", "cluster", "iterative"]),
            "content": rng.choice(["ramp", "opaque", "photo", "cutout"]), "width": w, "height": h,
            "aw": rng.random() < 0.25}
    if kind == "device":
        case["channels"] = 4
    return case


# ---------------------------------------------------------------------------
# contents

def _field(width, height, channels, gen, octaves=6):
    """Smooth multi-octave field in [0, 255], (height, width, channels) float."""
    out = torch.zeros((1, channels, height, width), device="cuda")
    total = 0.0
    for o in range(octaves):
        cells = 4 << o
        amp = 0.55 ** o
        total += amp
        grid = torch.rand((1, channels, cells + 1, cells + 1), generator=gen, device="cuda")
        out += amp * torch.nn.functional.interpolate(grid, size=(height, width), mode="bilinear", align_corners=True)
    return (out[0] * (255.0 / total)).permute(1, 2, 0)


def _image(content, width, height, channels, seed):
    """(height, width, channels) u8 image on the GPU."""
    if content in ("ramp", "opaque"):
        return workloads.ramp_texture_torch(width, height, seed, "cuda", alpha=content)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if content == "noise":
        used = 1 if channels == 1 else 2
        f = _field(width, height, used, gen)
        f = f + torch.randint(-3, 4, f.shape, generator=gen, device="cuda")
        f = f.round().clamp(0, 255).to(torch.uint8)
        if channels != 4:
            return f.contiguous()
        img = torch.zeros((height, width, 4), dtype=torch.uint8, device="cuda")
        img[..., :used] = f
        img[..., 3] = 255
        return img
    f = _field(width, height, 3, gen) * 1.6 - 76.0  # most of the range, some of it clipped
    f = f + torch.randint(0, 2, f.shape, generator=gen, device="cuda")
    img = torch.full((height, width, 4), 255, dtype=torch.uint8, device="cuda")
    img[..., :3] = f.round().clamp(0, 255).to(torch.uint8)
    if content == "cutout":
        m = _field(width, height, 1, gen, 5)[..., 0]
        img[..., 3] = ((m - 110.0) * 8.0).round().clamp(0, 255).to(torch.uint8)
    return img


def _params(case):
    return tx.Params(algorithm=tx.Algorithm(_ALG[case["alg"]]), weigh_colour_by_alpha=bool(case.get("aw", False)))


def _specs(n, min_side, max_side, formats, algorithms, spread):
    """Sizes, formats and algorithms of a set of textures: part of the case, not of the seed."""
    return workloads.batch_specs(n, seed=spread, min_side=min_side, max_side=max_side, formats=formats,
                                 algorithms=algorithms)


def _levels(width, height):
    out = [(width, height)]
    while width > 1 or height > 1:
        width, height = max(1, width // 2), max(1, height // 2)
        out.append((width, height))
    return out


# ---------------------------------------------------------------------------
# prepare / run

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "serve":
        return _prepare_serve(case, seed)
    fmt = tx.Format(_FMT[case["fmt"]])
    if kind == "block":
        img = _image(case["content"], 4, 4, 4, seed).cpu().numpy()
        return {"kind": kind, "fmt": fmt, "src": np.ascontiguousarray(img).reshape(64), "mask": case["mask"],
                "params": _params(case), "out": np.zeros(fmt.block_size(), np.uint8)}
    w, h = case["width"], case["height"]
    size = fmt.compressed_size(w, h)
    if kind == "host":
        img = np.ascontiguousarray(_image(case["content"], w, h, 4, seed).cpu().numpy())
        return {"kind": kind, "fmt": fmt, "src": img, "w": w, "h": h, "params": _params(case),
                "out": np.zeros(size, np.uint8)}
    channels = case.get("channels", 4)
    img = _image(case["content"], w, h, channels, seed)
    blocks = torch.zeros(size, dtype=torch.uint8, device="cuda")
    state = {"kind": kind, "fmt": fmt, "src": img, "w": w, "h": h, "channels": channels, "params": _params(case),
             "out": blocks}
    if kind == "decode":
        tx.compress_device(fmt, img.data_ptr(), w * channels, channels, w, h, state["params"], blocks.data_ptr(), size,
                           torch.cuda.current_stream().cuda_stream)
        state["src"] = blocks
        state["out"] = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    return state


def _prepare_batch(case, seed):
    specs = _specs(case["textures"], case["min_side"], case["max_side"], (0, 2, 4), (0, 1, 2), case["spread"])
    kinds = ("ramp", "photo", "cutout")
    # all mip levels live in one buffer and all compressed levels in another, as in an asset package
    pad = lambda n: (n + 15) // 16 * 16
    dims = [(tx.Format(s["format"]), _levels(s["width"], s["height"])) for s in specs]
    mips = torch.zeros(sum(pad(w * h * 4) for _, lv in dims for w, h in lv[1:]) + 16, dtype=torch.uint8, device="cuda")
    out = torch.zeros(sum(pad(f.compressed_size(w, h)) for f, lv in dims for w, h in lv), dtype=torch.uint8,
                      device="cuda")
    base, jobs, items = [], [], []  # jobs[d]: the mip jobs that make level d + 1 of every texture
    m = o = 0
    for t, (s, (fmt, lv)) in enumerate(zip(specs, dims)):
        img = _image(kinds[t % 3], s["width"], s["height"], 4, seed * 1009 + t)
        base.append(img)
        prm = tx.Params(algorithm=tx.Algorithm(s["algorithm"]))
        src = img.data_ptr()
        for d, (w, h) in enumerate(lv):
            if d:
                sw, sh = lv[d - 1]
                dst = mips.data_ptr() + m
                m += pad(w * h * 4)
                while len(jobs) < d:
                    jobs.append([])
                jobs[d - 1].append((src, sw * 4, sw, sh, 4, dst, w * 4))
                src = dst
            items.append(tx.batch_item(fmt, src, w * 4, w, h, prm, out.data_ptr() + o))
            o += pad(fmt.compressed_size(w, h))
    return {"kind": "batch", "jobs": jobs, "plan": tx.Batch(items), "base": base, "mips": mips, "out": out}


def _prepare_serve(case, seed):
    specs = _specs(case["requests"], case["min_side"], case["max_side"], (0, 2, 4), (2,), case["spread"])
    reqs = []
    kinds = ("photo", "ramp", "cutout")
    for t, s in enumerate(specs):
        img = _image(kinds[t % 3], s["width"], s["height"], 4, seed * 1009 + t)
        out = np.zeros(tx.chain_compressed_size(s["format"], s["width"], s["height"], True), np.uint8)
        reqs.append((np.ascontiguousarray(img.cpu().numpy()), s["width"], s["height"], s["format"],
                     tx.Params(algorithm=tx.Algorithm(s["algorithm"])), out))
    return {"kind": "serve", "server": tx.Server(memory_budget=2 << 30), "reqs": reqs}


def run(state):
    kind = state["kind"]
    if kind == "block":
        state["fmt"].compress_block_masked(state["src"], state["mask"], state["params"], state["out"])
        return state["out"]
    if kind == "host":
        state["fmt"].compress(state["src"], state["w"], state["h"], state["params"], state["out"])
        return state["out"]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(img, w, h, fmt, prm, out) for img, w, h, fmt, prm, out in state["reqs"]]
        for rid in ids:
            server.wait(rid)
        return [r[5] for r in state["reqs"]]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "batch":
        for jobs in state["jobs"]:
            tx.mip_batch_device(jobs, stream)
        state["plan"].launch(stream)
        return [state["out"], state["mips"]]
    if kind == "decode":
        src, out = state["src"], state["out"]
        tx.decompress_device(state["fmt"], src.data_ptr(), src.numel(), state["w"], state["h"], out.data_ptr(),
                             state["w"] * 4, stream)
        return out
    src, out = state["src"], state["out"]
    tx.compress_device(state["fmt"], src.data_ptr(), state["w"] * state["channels"], state["channels"], state["w"],
                       state["h"], state["params"], out.data_ptr(), out.numel(), stream)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without

# Operations per block, counted from the algorithms' definitions: a colour fit
# forms the centroid and covariance of 16 points (22 per point), the power
# iteration (8 x 20) and the projections (5 per point); the range fit then
# measures 16 points against 4 codes (8 each); the cluster fit weighs 967
# partitions of the ordered points in 3 channels (151 more for BC1's
# three-colour form), about 8 operations each; the alpha search compares 16
# values with two books of 8 codes (2 each).
_FIT = 16 * 22 + 8 * 20 + 16 * 5
_ALPHA = 16 * 16 * 2


def _block_flops(fmt, alg):
    if fmt == "bc4":
        return _ALPHA
    if fmt == "bc5":
        return 2 * _ALPHA
    n = _FIT + (_ALPHA if fmt == "bc3" else 0)
    if alg == "range":
        return n + 16 * 4 * 8 * (2 if fmt == "bc1" else 1)
    return n + 8 * (967 + (151 if fmt == "bc1" else 0))


def _image_work(fmt, alg, w, h, channels):
    nb = ((w + 3) // 4) * ((h + 3) // 4)
    return w * h * channels + nb * (8 if fmt in ("bc1", "bc4") else 16), nb * _block_flops(fmt, alg)


def work(case):
    kind = case["kind"]
    if kind == "block":
        b, f = _image_work(case["fmt"], case["alg"], 4, 4, 4)
        return {"bytes": b, "flops": f}
    if kind == "decode":
        b, _ = _image_work(case["fmt"], "range", case["width"], case["height"], 4)
        return {"bytes": b, "flops": 0}
    if kind in ("batch", "serve"):
        if kind == "batch":
            specs = _specs(case["textures"], case["min_side"], case["max_side"], (0, 2, 4), (0, 1, 2), case["spread"])
        else:
            specs = _specs(case["requests"], case["min_side"], case["max_side"], (0, 2, 4), (2,), case["spread"])
        names = {v: k for k, v in _FMT.items()}
        algs = {v: k for k, v in _ALG.items()}
        nbytes = flops = 0
        for s in specs:
            for d, (w, h) in enumerate(_levels(s["width"], s["height"])):
                b, f = _image_work(names[s["format"]], algs[s["algorithm"]], w, h, 4)
                nbytes += b + (w * h * 4 if d and kind == "batch" else 0)  # a batch hands its mip levels out too
                flops += f
        return {"bytes": nbytes, "flops": flops}
    b, f = _image_work(case["fmt"], case["alg"], case["width"], case["height"], case.get("channels", 4))
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """Every output is bytes (blocks, pixels, mip levels), equal or not: no 64-bit value stands behind them."""
    return None
