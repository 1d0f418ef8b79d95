"""The work whose speed counts: passes through the package's public calls, from one small image to
a batch of textures of mixed sizes and formats.

listed() are fixed sizes, draw() gives more of the same ranges. prepare() makes what a program has
in hand before the call (textures from texgen's seeded generators, .crn files, a network, a batch
plan), run() is one pass and returns the pass's whole outputs.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import crunch2_gb300 as cg
from crunch2_gb300 import learned, texgen

FORMATS = {"dxt1": cg.FMT_DXT1, "dxt5": cg.FMT_DXT5, "dxn": cg.FMT_DXN_XY, "dxt5a": cg.FMT_DXT5A}
COLOUR, BOTH = cg.FLAG_PERCEPTUAL, cg.FLAG_USE_BOTH_BLOCK_TYPES

# The reference search's candidate x unique-colour evaluations of a DXT1 block (200,060,536 over the
# 87,383 blocks of a 1024x1024 chain), 27 operations each. The alpha search has no such count: its
# least work depends on the method, so alpha elements are counted by their bytes alone.
DXT1_FLOPS = 200060536 / 87383 * 27
MLP_FLOPS = 2 * (48 * 256 + 256 * 256 + 256 * 7)


def listed():
    return [
        # one small sprite or UI image handed to the plain encoder: launches and latency
        {"name": "encode_dxt1_64", "kind": "image", "w": 64, "h": 64, "fmt": "dxt1", "host": False, "quality": 4},
        # a 1024x1024 colour texture with its mip chain as blocks on the device (the bench's workload)
        {"name": "encode_dxt1_chain_1024", "kind": "blocks", "w": 1024, "h": 1024, "perceptual": True, "quality": 4},
        # a screenshot-sized image with alpha, sides no multiple of 4, in host memory
        {"name": "encode_dxt5_ragged", "kind": "image", "w": 1021, "h": 683, "fmt": "dxt5", "host": True, "quality": 4},
        # a 2048x2048 normal map: two alpha searches per block, no colour
        {"name": "encode_dxn_2048", "kind": "image", "w": 2048, "h": 2048, "fmt": "dxn", "host": False, "quality": 4},
        # a build step's textures of uneven sizes (powers of two 32..2048) and mixed formats, one plan
        {"name": "encode_batch_24", "kind": "encode_batch", "textures": 24, "most": 2048, "set": 3000},
        # the learned proposal on a 1024x1024 chain
        {"name": "learned_chain_1024", "kind": "learned", "w": 1024, "h": 1024, "quality": 3},
        # one training step of the proposal network at its training batch
        {"name": "train_8192", "kind": "train", "batch": 8192, "tau": 0.75},
        # a game loading one 1024x1024 .crn: open, all levels to device memory, close
        {"name": "unpack_dxt1_1024", "kind": "unpack", "w": 1024, "h": 1024, "fmt": "dxt1", "quality": 128, "host": False},
        # a level load: files of uneven sizes and mixed formats transcoded by one plan
        {"name": "unpack_batch_24", "kind": "unpack_batch", "textures": 24, "most": 2048, "set": 3000},
        # an asset pipeline writing one 1024x1024 .crn at the default quality
        {"name": "crn_dxt1_1024", "kind": "crn", "w": 1024, "h": 1024, "fmt": "dxt1", "quality": 128},
        # the same for an odd-sized image with alpha at a higher quality
        {"name": "crn_dxt5_ragged", "kind": "crn", "w": 333, "h": 180, "fmt": "dxt5", "quality": 192},
        # crunch's default mip generation of a large texture
        {"name": "mips_4096", "kind": "mips", "w": 4096, "h": 4096, "filter": "kaiser", "scale": 0.9, "srgb": True,
         "wrap": False, "alpha": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["blocks", "image", "image", "encode_batch", "learned", "train", "unpack", "unpack",
                       "unpack_batch", "crn", "crn", "mips", "mips"])
    quality = rng.choice([4, 4, 4, 3, 2, 1])
    fmt = rng.choice(["dxt1", "dxt1", "dxt5", "dxn", "dxt5a"])
    if kind == "blocks":
        return {"kind": kind, "w": _log(rng, 4, 1024), "h": _log(rng, 4, 1024), "perceptual": rng.random() < 0.75,
                "quality": quality}
    if kind == "image":
        return {"kind": kind, "w": _log(rng, 4, 1500), "h": _log(rng, 4, 1500), "fmt": fmt,
                "host": rng.random() < 0.4, "quality": quality}
    if kind in ("encode_batch", "unpack_batch"):
        return {"kind": kind, "textures": _log(rng, 3, 24), "most": rng.choice([512, 1024]), "set": rng.randrange(1 << 20)}
    if kind == "learned":
        return {"kind": kind, "w": _log(rng, 16, 1024), "h": _log(rng, 16, 1024), "quality": rng.choice([3, 3, 4, 2])}
    if kind == "train":
        return {"kind": kind, "batch": _log(rng, 256, 8192), "tau": rng.choice([0.75, 0.0])}
    if kind == "unpack":
        return {"kind": kind, "w": _log(rng, 16, 1024), "h": _log(rng, 16, 1024), "fmt": fmt,
                "quality": rng.choice([64, 128, 192, 255]), "host": rng.random() < 0.5}
    if kind == "crn":
        return {"kind": kind, "w": _log(rng, 32, 800), "h": _log(rng, 32, 800), "fmt": fmt,
                "quality": rng.choice([32, 128, 192, 255])}
    return {"kind": kind, "w": _log(rng, 16, 4096), "h": _log(rng, 16, 4096),
            "filter": rng.choice(["kaiser", "kaiser", "box", "tent", "lanczos4", "mitchell"]),
            "scale": rng.choice([0.9, 0.9, 1.0, 1.2]), "srgb": rng.random() < 0.75, "wrap": rng.random() < 0.3,
            "alpha": rng.random() < 0.6}


def _dims(w, h):
    return [(max(1, w >> l), max(1, h >> l)) for l in range(max(w, h).bit_length())]


def _chain_blocks(w, h):
    return sum(((a + 3) // 4) * ((b + 3) // 4) for a, b in _dims(w, h))


def _chain_bytes(w, h):
    return 4 * sum(a * b for a, b in _dims(w, h))


def _members(case):
    """(width, height, format) of a batch's textures: sides from the powers of two 32..most, 60 %
    DXT1, 25 % DXT5, 15 % DXN."""
    r = random.Random(case["set"])
    sides = [1 << i for i in range(5, case["most"].bit_length())]
    return [(r.choice(sides), r.choice(sides), r.choices(["dxt1", "dxt5", "dxn"], [60, 25, 15])[0])
            for _ in range(case["textures"])]


def _texture(w, h, fmt, seed):
    if fmt == "dxn":
        return texgen.normal_map_torch(w, h, seed)
    return texgen.colour_texture_torch(w, h, seed, with_alpha_noise=fmt != "dxt1")


def _blocks(img):
    """The edge-clamped 4x4 blocks of an image of any size."""
    h, w = img.shape[:2]
    ys = torch.arange((h + 3) // 4 * 4, device=img.device).clamp(max=h - 1)
    xs = torch.arange((w + 3) // 4 * 4, device=img.device).clamp(max=w - 1)
    return texgen.image_blocks_torch(img[ys][:, xs].contiguous())


def _chain(w, h, fmt, seed):
    return texgen.mip_chain_torch(_texture(w, h, fmt, seed))


def _host_chain(w, h, fmt, seed):
    return [[np.ascontiguousarray(l.cpu().numpy()) for l in _chain(w, h, fmt, seed)]]


def _targets(batch, seed):
    """Endpoints in [0, 1] and a small error bound, unrelated to the blocks: residuals as large as
    those of training's beginning."""
    g = torch.Generator().manual_seed(seed)
    t = torch.rand((batch, 8), generator=g)
    t[:, 6] *= 0.2
    t[:, 7] = 0
    return t


def _train_inputs(case, seed):
    side = 4 * math.ceil(math.sqrt(case["batch"]))
    blocks = texgen.image_blocks_torch(texgen.colour_texture_torch(side, side, seed))[:case["batch"]]
    return blocks.contiguous(), _targets(case["batch"], seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "image":
        img = _texture(case["w"], case["h"], case["fmt"], seed)
        return {"case": case, "img": img.cpu().numpy() if case["host"] else img}
    if kind == "blocks":
        return {"case": case, "blocks": torch.cat([_blocks(l) for l in _chain(case["w"], case["h"], "dxt1", seed)])}
    if kind == "encode_batch":
        items = []
        for i, (w, h, fmt) in enumerate(_members(case)):
            rgba = torch.cat([l.reshape(-1) for l in _chain(w, h, fmt, seed * 64 + i)])
            f = FORMATS[fmt]
            out = torch.empty(_chain_blocks(w, h) * cg.bytes_per_block(f), dtype=torch.uint8, device="cuda")
            items.append((rgba, out, w, h, len(_dims(w, h)), f))
        return {"case": case, "batch": cg.EncodeBatch(items), "outs": [it[1] for it in items]}
    if kind == "learned":
        return {"case": case, "net": learned.default_net(),
                "blocks": torch.cat([_blocks(l) for l in _chain(case["w"], case["h"], "dxt1", seed)])}
    if kind == "train":
        net = learned.default_net()
        if case["tau"] > 0:
            net.set_bound_loss(case["tau"], 0.25)
        blocks, targets = _train_inputs(case, seed)
        return {"case": case, "net": net, "blocks": blocks, "targets": targets.cuda()}
    if kind == "unpack":
        return {"case": case, "file": cg.compress_crn(_host_chain(case["w"], case["h"], case["fmt"], seed),
                                                      FORMATS[case["fmt"]], case["quality"])}
    if kind == "unpack_batch":
        members = _members(case)
        files = cg.compress_crn_batch([(_host_chain(w, h, fmt, seed * 64 + i), FORMATS[fmt], 128, COLOUR)
                                       for i, (w, h, fmt) in enumerate(members)], threads=8)
        ctxs = [cg.unpack_begin(f) for f in files]
        outs = [torch.empty(sum(c.level_bytes(l) for l in range(c.levels)), dtype=torch.uint8, device="cuda") for c in ctxs]
        return {"case": case, "batch": cg.UnpackBatch([(c, 0, c.levels, o) for c, o in zip(ctxs, outs)]), "outs": outs}
    if kind == "crn":
        return {"case": case, "faces": _host_chain(case["w"], case["h"], case["fmt"], seed)}
    if kind == "mips":
        return {"case": case, "img": _texture(case["w"], case["h"], "dxt5" if case["alpha"] else "dxt1", seed)}
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "image":
        return cg.compress_image(state["img"], FORMATS[case["fmt"]], COLOUR | BOTH, quality=case["quality"])
    if kind == "blocks":
        return cg.dxt1_optimize(state["blocks"], case["perceptual"], True, with_error=True, quality=case["quality"])
    if kind in ("encode_batch", "unpack_batch"):
        state["batch"].launch(use_graph=True)
        return state["outs"]
    if kind == "learned":
        return state["net"].encode(state["blocks"], fallback_quality=case["quality"])
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["blocks"], state["targets"])
        return [loss] + [net.get(i, grad=True) for i in range(len(learned.PARAM_SHAPES))]
    if kind == "unpack":
        with cg.unpack_begin(state["file"]) as ctx:
            out = None
            if not case["host"]:
                total = sum(ctx.level_bytes(l) for l in range(ctx.levels))
                out = torch.empty(total, dtype=torch.uint8, device="cuda")
            return ctx.unpack_levels(out=out)
    if kind == "crn":
        data = np.frombuffer(cg.compress_crn(state["faces"], FORMATS[case["fmt"]], case["quality"]), np.uint8)
        whole = np.zeros(_crn_most(case), np.uint8)  # one length for every texture: files differ in size
        whole[:data.size] = data
        return {"size": data.size, "file": whole}
    if kind == "mips":
        return cg.generate_mipmaps(state["img"], case["filter"], case["scale"], case["srgb"], case["wrap"], case["alpha"])
    raise ValueError(kind)


def _file_bytes(blocks, fmt):
    """About what a .crn holds per block: 1.1 bits a texel for DXT1, 2 for DXT5 and DXN."""
    return int(blocks * 16 * (2.0 if fmt in ("dxt5", "dxn") else 1.1) / 8)


def _crn_most(case):
    """No .crn of the case is larger: its blocks as they are, and the palettes."""
    return _chain_blocks(case["w"] + 8, case["h"] + 8) * 16 + (1 << 18)


def work(case):
    kind = case["kind"]
    colour = lambda fmt: DXT1_FLOPS if fmt in ("dxt1", "dxt5") else 0
    bpb = lambda fmt: 16 if fmt in ("dxt5", "dxn") else 8
    if kind == "image":
        n = ((case["w"] + 3) // 4) * ((case["h"] + 3) // 4)
        full = case["quality"] == 4
        return {"bytes": case["w"] * case["h"] * 4 + n * bpb(case["fmt"]), "flops": n * colour(case["fmt"]) * full}
    if kind == "blocks":
        n = _chain_blocks(case["w"], case["h"])
        return {"bytes": n * (64 + 8 + 8), "flops": n * DXT1_FLOPS * (case["quality"] == 4)}
    if kind == "encode_batch":
        m = [(_chain_bytes(w, h), _chain_blocks(w, h), f) for w, h, f in _members(case)]
        return {"bytes": sum(b + n * bpb(f) for b, n, f in m), "flops": sum(n * colour(f) for _, n, f in m)}
    if kind == "learned":
        n = _chain_blocks(case["w"], case["h"])
        return {"bytes": n * (64 + 8), "flops": n * MLP_FLOPS}
    if kind == "train":
        params = sum(math.prod(s) for s in learned.PARAM_SHAPES)
        return {"bytes": case["batch"] * (64 + 32) + params * 4 * 7, "flops": 3 * case["batch"] * MLP_FLOPS}
    if kind in ("unpack", "unpack_batch"):
        m = [(case["w"], case["h"], case["fmt"])] if kind == "unpack" else _members(case)
        return {"bytes": sum(_chain_blocks(w, h) * bpb(f) + _file_bytes(_chain_blocks(w, h), f) for w, h, f in m), "flops": 0}
    if kind == "crn":
        return {"bytes": _chain_bytes(case["w"], case["h"]) + _file_bytes(_chain_blocks(case["w"], case["h"]), case["fmt"]),
                "flops": 0}
    # mips: a level's row pass reads all of level 0, its taps spread over the filter's support; each
    # tap is a multiply and an add on four channels, none of them sharable between levels
    support = {"box": 0.5, "tent": 1.0, "lanczos4": 4.0, "mitchell": 2.0, "kaiser": 3.0}[case["filter"]]
    taps = max(1.0, 2 * support * case["scale"])
    flops = 0
    for a, b in _dims(case["w"], case["h"])[1:]:
        flops += 8 * taps * (case["w"] * case["h"] + a * case["h"])
    return {"bytes": case["w"] * case["h"] * 4 + _chain_bytes(case["w"], case["h"]), "flops": flops}


def exact(case, seed):
    """The loss and gradients of a training step in 64 bits; every other output is whole bytes."""
    if case["kind"] != "train":
        return None
    blocks, targets = _train_inputs(case, seed)
    p = {k: v.astype(np.float64) for k, v in np.load(learned.WEIGHTS).items()}
    t = targets.numpy().astype(np.float64)[:, :7]
    x = blocks.cpu().numpy().reshape(-1, 16, 4)[:, :, :3].reshape(-1, 48) / 255.0
    c, k = math.sqrt(2 / math.pi), 0.044715

    def act(a):
        th = np.tanh(c * (a + k * a ** 3))
        return 0.5 * a * (1 + th), 0.5 * (1 + th) + 0.5 * a * (1 - th * th) * c * (1 + 3 * k * a * a)

    h1, s1 = act(x @ p["W1"].T + p["b1"])
    h2, s2 = act(h1 @ p["W2"].T + p["b2"])
    y = h2 @ p["W3"].T + p["b3"]
    n = case["batch"]
    d = y[:, :7] - t
    dy = np.zeros_like(y)
    dy[:, :7] = 2 * d / n
    loss = (d[:, :6] ** 2).sum()
    if case["tau"] > 0:
        tau, r = case["tau"], d[:, 6]
        loss += (0.25 * np.where(r > 0, (1 - tau) * r, -tau * r)).sum()
        dy[:, 6] = 0.25 * np.where(r > 0, 1 - tau, -tau) / n
    else:
        loss += (d[:, 6] ** 2).sum()
    d2 = (dy @ p["W3"]) * s2
    d1 = (d2 @ p["W2"]) * s1
    return [loss / n, d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0)]
