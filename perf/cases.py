"""The encoder's timed workloads, each through the package's public entry points.

A case is one call (or one flow of calls) that a program with textures to
compress makes: encodes of device-resident textures, of host images and of
loose 4x4 cells, a batch, a request loop, and the steps around the encode
(padding, outline mask, decode, glitch and partition maps).  The presets are
the ones the command-line flags select: ``draft``, ``default``, ``precise``
(kDenoise 0), ``slow`` and ``data`` (linear weights, for normal maps and other
non-colour data), and ``m6i2`` (the Mode6Index2 pass alone).

Images are made on the GPU from the seed, with the distributions of
``nebc7_gb300.synth``: ``photo`` (four octaves of correlated value noise and
hard-edged polygons), ``alpha`` (a gradient with value noise, about 30 % of the
pixels transparent in blobs, 15 % on a ramp) and ``normals`` (unit normals of a
height field, opaque).
"""

import math

import numpy as np
import torch
import torch.nn.functional as F

import nebc7_gb300 as nb
from nebc7_gb300._native import Settings, check

PRESETS = {
    # name: (kDenoise, step, draft, normal, slow, linear)
    "m6i2": (1, 9, 2, 0, 0, 0),
    "draft": (1, 9, 1, 0, 0, 0),
    "default": (1, 9, 1, 1, 0, 0),
    "precise": (0, 0, 1, 1, 0, 0),
    "slow": (1, 9, 1, 1, 1, 0),
    "data": (1, 9, 1, 1, 0, 1),
}

# Integer operations of the reference's own search per 4x4 block (table terms
# and error terms, counted on images like these), the least that an exact
# encode has to decide with.
OPS_PER_BLOCK = {"m6i2": 1.2e3, "draft": 2.5e3, "default": 4.6e5, "precise": 1.8e6, "slow": 5.9e6, "data": 2.6e6}


def listed():
    return [
        # 256 loose cells with masks through the block API: the job that the
        # reference's worker pool hands to its block kernel; latency counts.
        {"name": "cells256_default", "do": "cells", "image": "alpha", "preset": "default", "n": 256},
        # One small texture (a UI icon) already on the device.
        {"name": "icon64_default", "do": "device", "image": "photo", "preset": "default", "w": 64, "h": 64, "mask": False,
         "start": False, "stats": False},
        # The command-line's default run on an ordinary opaque texture.
        {"name": "photo1024_default", "do": "device", "image": "photo", "preset": "default", "w": 1024, "h": 1024,
         "mask": False, "start": False, "stats": False},
        # /draft on a large texture: previews and build farms.
        {"name": "photo4096_draft", "do": "device", "image": "photo", "preset": "draft", "w": 4096, "h": 4096, "mask": False,
         "start": False, "stats": False},
        # The precise preset with its quality report, as a final asset build runs it.
        {"name": "photo1024_precise", "do": "device", "image": "photo", "preset": "precise", "w": 1024, "h": 1024,
         "mask": False, "start": False, "stats": True},
        # /slow on a sprite sheet with transparency and its outline mask: the longest search.
        {"name": "alpha1024_slow", "do": "device", "image": "alpha", "preset": "slow", "w": 1024, "h": 1024, "mask": True,
         "start": False, "stats": False},
        # /data on a small normal map (linear weights).
        {"name": "normals256_data", "do": "device", "image": "normals", "preset": "data", "w": 256, "h": 256, "mask": False,
         "start": False, "stats": False},
        # A host image of odd size with transparency through the command-line's
        # whole encode path: padding, mask, copies, encode, report sums.
        {"name": "sprite1118x1105_default", "do": "image", "image": "alpha", "flags": "", "denoise": 1, "step": 9, "w": 1118,
         "h": 1105},
        # Incremental re-encode: a texture whose kept blocks came from a draft run.
        {"name": "alpha1000x516_restart", "do": "device", "image": "alpha", "preset": "default", "w": 1000, "h": 516,
         "mask": True, "start": True, "stats": False},
        # A batch of textures of mixed sizes and presets under one kept plan.
        {"name": "batch24_mixed", "do": "batch", "n": 24, "lo": 4, "hi": 512},
        # The driver's steps around an encode of a large texture, on the device:
        # padding and outline mask, decode, glitch map, partition map.
        {"name": "tools4093x4090", "do": "tools", "image": "alpha", "w": 4093, "h": 4090, "radius": 1},
        # The request loop: textures of mixed sizes and presets submitted together from host memory.
        {"name": "serve24_mixed", "do": "serve", "n": 24, "lo": 64, "hi": 512},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["cells", "device", "device", "device", "device", "image", "batch", "tools", "serve"])
    if do == "cells":
        return {"do": do, "image": rng.choice(["photo", "alpha"]), "preset": rng.choice(["draft", "default", "precise"]),
                "n": _side(rng, 1, 8192)}
    if do == "device":
        preset = rng.choice(["m6i2", "draft", "default", "default", "precise", "slow", "data"])
        most = {"m6i2": 4096, "draft": 4096, "default": 2048, "precise": 1024, "slow": 768, "data": 256}[preset]
        w, h = (4 * max(1, _side(rng, 4, most) // 4) for _ in range(2))
        image = "normals" if preset == "data" else rng.choice(["photo", "alpha"])
        return {"do": do, "image": image, "preset": preset, "w": w, "h": h, "mask": image == "alpha" and rng.random() < 0.75,
                "start": rng.random() < 0.25, "stats": rng.random() < 0.25}
    if do == "image":
        flags, denoise, step, most = rng.choice([("/draft", 1, 9, 2048), ("", 1, 9, 1536), ("/retina", 1, 9, 1536),
                                                 ("/nomask", 0, 0, 768), ("/slow", 1, 9, 512)])
        return {"do": do, "image": rng.choice(["photo", "alpha"]), "flags": flags, "denoise": denoise, "step": step,
                "w": _side(rng, 1, most), "h": _side(rng, 1, most)}
    if do == "batch":
        return {"do": do, "n": rng.randint(2, 40), "lo": 4, "hi": rng.choice([64, 128, 256, 512])}
    if do == "tools":
        return {"do": do, "image": rng.choice(["photo", "alpha"]), "w": _side(rng, 1, 4096), "h": _side(rng, 1, 4096),
                "radius": rng.choice([-1, 1, 2])}
    return {"do": do, "n": rng.randint(1, 32), "lo": 16, "hi": rng.choice([64, 128, 256, 512])}


# ---- images ---------------------------------------------------------------


def _gen(seed):
    return torch.Generator().manual_seed(int(seed) & 0x7FFFFFFF)


def _ints(g, lo, hi, *shape):
    """Integers in [lo, hi], drawn on the host (the same on every device)."""
    return torch.randint(lo, hi + 1, shape, generator=g)


def _noise(g, n, w, h, cell, amp):
    """n planes of bilinear value noise in [-amp, amp], int32[n, h, w]."""
    lat = _ints(g, -amp, amp, 1, n, h // cell + 2, w // cell + 2).float().cuda()
    up = F.interpolate(lat, scale_factor=float(cell), mode="bilinear", align_corners=False)
    return up[0, :, cell // 2:cell // 2 + h, cell // 2:cell // 2 + w].round().int()


def _fine(seed, lo, hi, *shape):
    """Per-pixel noise in [lo, hi], made on the device."""
    return torch.randint(lo, hi + 1, shape, generator=torch.Generator("cuda").manual_seed(int(seed) & 0x7FFFFFFF),
                         device="cuda", dtype=torch.int32)


def _polygons(g, rgb, count):
    _, h, w = rgb.shape
    top = max(8, min(w, h) // 6)
    for _ in range(count):
        cx, cy = int(_ints(g, 0, w - 1, 1)), int(_ints(g, 0, h - 1, 1))
        r, k = int(_ints(g, 4, top, 1)), int(_ints(g, 3, 6, 1))
        a = torch.sort(_ints(g, 0, 63, k))[0].tolist()
        colour = _ints(g, 0, 255, 3, 1, 1).int().cuda(non_blocking=True)
        p = [(cx + r * math.cos(t * math.pi / 32), cy + r * math.sin(t * math.pi / 32)) for t in a]
        x0, x1 = max(0, cx - r), min(w, cx + r + 1)
        y0, y1 = max(0, cy - r), min(h, cy + r + 1)
        ys = torch.arange(y0, y1, device="cuda").float()[:, None]
        xs = torch.arange(x0, x1, device="cuda").float()[None, :]
        inside = None
        for (ax, ay), (bx, by) in zip(p, p[1:] + p[:1]):
            e = (bx - ax) * (ys - ay) - (by - ay) * (xs - ax) >= 0
            inside = e if inside is None else inside & e
        part = rgb[:, y0:y1, x0:x1]
        part.copy_(torch.where(inside, colour, part))


def _gradient(g, w, h):
    c = _ints(g, 0, 255, 1, 3, 2, 2).float().cuda()
    return F.interpolate(c, size=(h, w), mode="bilinear", align_corners=True)[0].round().int()


def _image(kind, w, h, seed):
    """uint8[h, w, 4] BGRA on the GPU."""
    g = _gen(seed)
    alpha = None
    if kind == "photo":
        rgb = _ints(g, 64, 192, 3, 1, 1).int().cuda().expand(3, h, w).clone()
        for cell, amp in ((64, 96), (32, 48), (16, 24), (8, 12)):
            rgb += ((2 * _noise(g, 1, w, h, cell, amp) + _noise(g, 3, w, h, cell, amp)) * 229) >> 9
        _polygons(g, rgb, max(4, min(200, w * h // 5000)))
        rgb += _fine(seed, -1, 1, 3, h, w)
    elif kind == "alpha":
        rgb = _gradient(g, w, h) + _noise(g, 3, w, h, 8, 40) + _fine(seed, -3, 3, 3, h, w)
        field = (_noise(g, 1, w, h, max(8, min(w, h) // 8), 1000) + _noise(g, 1, w, h, max(4, min(w, h) // 32), 250))[0]
        flat = torch.sort(field.flatten()[:: max(1, w * h // 65536)])[0]
        t0, t1 = flat[flat.numel() * 30 // 100], flat[flat.numel() * 45 // 100]
        clear, ramp = field < t0, (field >= t0) & (field < t1)
        alpha = torch.where(ramp, 1 + (field - t0) * 253 // torch.clamp(t1 - t0, min=1), torch.full_like(field, 255))
        alpha = torch.where(clear, torch.zeros_like(alpha), alpha)
        rgb = torch.where(clear, _fine(seed + 1, 0, 255, 3, h, w), rgb)
    else:
        z = sum(_noise(g, 1, w + 1, h + 1, cell, amp)[0] for cell, amp in ((32, 256), (8, 48)))
        nx, ny = (z[:-1, :-1] - z[:-1, 1:]).float() / 32, (z[:-1, :-1] - z[1:, :-1]).float() / 32
        inv = 1 / torch.sqrt(1 + nx * nx + ny * ny)
        rgb = torch.stack([nx * inv, ny * inv, inv]).mul_(127.5).add_(127.5).round_().int() + _fine(seed, -1, 1, 3, h, w)
    out = torch.full((h, w, 4), 255, dtype=torch.uint8, device="cuda")
    out[:, :, :3] = rgb.clamp_(0, 255).flip(0).permute(1, 2, 0).byte()
    if alpha is not None:
        out[:, :, 3] = alpha.byte()
    return out


def _outline(bgra):
    """The alpha outline mask of radius 1 (bytes A, G, R, B per pixel)."""
    on = F.max_pool2d((bgra[None, None, :, :, 3] != 0).float(), 3, 1, 1)[0, 0] > 0
    mask = torch.full_like(bgra, 255)
    mask[:, :, 1:] = (on.byte() * 255)[:, :, None]
    return mask


def _settings(preset):
    return Settings(*PRESETS[preset])


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _encode(dst, bgra, mask, preset, stats=False):
    d, s, draft, normal, slow, linear = PRESETS[preset]
    h, w = bgra.shape[:2]
    return nb.encode_device(dst.data_ptr(), bgra.data_ptr(), mask.data_ptr() if mask is not None else None, w * 4, w, h,
                            nb.Preset(d, s), draft, bool(normal), bool(slow), bool(linear), _stream(), stats)


def _blocks(w, h):
    return torch.zeros(((h // 4) * (w // 4), 16), dtype=torch.uint8, device="cuda")


# ---- the cases ------------------------------------------------------------


def _texture_list(case, seed, presets):
    """n textures (w, h, image kind, preset): sides log-uniform in [lo, hi]
    rounded up to x4, 60 % opaque, presets by the given shares.  Sizes and
    presets depend on the case alone, so that every seed is the same work."""
    g = _gen(1000 + case["n"])
    octaves = math.log2(case["hi"] / case["lo"])
    out = []
    for i in range(case["n"]):
        w, h = (min(case["hi"], (int(case["lo"] * 2 ** (octaves * float(torch.rand(1, generator=g)))) + 3) & ~3) for _ in range(2))
        kind = "alpha" if int(_ints(g, 0, 99, 1)) < 40 else "photo"
        roll = int(_ints(g, 0, 99, 1))
        preset = next(p for p, below in presets if roll < below)
        out.append((w, h, kind, preset, seed * 1000 + i))
    return out


BATCH_MIX = (("draft", 33), ("default", 66), ("precise", 100))
SERVE_MIX = (("default", 50), ("draft", 80), ("precise", 95), ("m6i2", 100))


def prepare(case, seed):
    do = case["do"]
    if do == "cells":
        n = case["n"]
        w = 4 * min(n, 64)
        h = 4 * -(-n // min(n, 64))
        img = _image(case["image"], max(w, 64), max(h, 64), seed)
        mask = _outline(img) if case["image"] == "alpha" else torch.full_like(img, 255)

        def cells(t):
            t = t[:h, :w].reshape(h // 4, 4, w // 4, 16).permute(0, 2, 1, 3)
            return t.reshape(-1, 64)[:n].contiguous().cpu().numpy()

        d, s, draft, normal, slow, linear = PRESETS[case["preset"]]
        core = nb.Bc7Core(nb.Preset(d, s))
        core.init_tables(draft, normal, slow, linear)
        return {"do": do, "core": core, "cells": cells(img), "masks": cells(mask), "blocks": np.zeros((n, 16), np.uint8)}
    if do == "device":
        img = _image(case["image"], case["w"], case["h"], seed)
        mask = _outline(img) if case["mask"] else None
        dst = _blocks(case["w"], case["h"])
        start = None
        if case["start"]:
            start = torch.zeros_like(dst)
            _encode(start, img, mask, "draft")
        check(nb.load().nebc7_init_device(PRESETS[case["preset"]][0]), "init")
        return {"do": do, "dst": dst, "bgra": img, "mask": mask, "start": start, "preset": case["preset"], "stats": case["stats"]}
    if do == "image":
        return {"do": do, "img": _image(case["image"], case["w"], case["h"], seed).cpu().numpy(), "flags": case["flags"],
                "preset": nb.Preset(case["denoise"], case["step"])}
    if do == "batch":
        keep, textures = [], []
        for w, h, kind, preset, s in _texture_list(case, seed, BATCH_MIX):
            img = _image(kind, w, h, s)
            mask = _outline(img) if kind == "alpha" else None
            dst = _blocks(w, h)
            keep.append((img, mask, dst))
            textures.append(nb.BatchTexture(dst.data_ptr(), img.data_ptr(), mask.data_ptr() if mask is not None else None,
                                            w * 4, w, h, _settings(preset)))
        return {"do": do, "keep": keep, "batch": nb.Batch(textures, from_scratch=True)}
    if do == "tools":
        w, h = case["w"], case["h"]
        src = _image(case["image"], w, h, seed)
        pw, ph = nb.padded_size(w, h)
        padded, mask, dec, bad = (torch.empty((ph, pw, 4), dtype=torch.uint8, device="cuda") for _ in range(4))
        blocks = _blocks(pw, ph)
        check(nb.load().nebc7_prepare_device(src.data_ptr(), w * 4, w, h, padded.data_ptr(), mask.data_ptr(), case["radius"],
                                             _stream()), "prepare")
        _encode(blocks, padded, mask, "draft")
        return {"do": do, "src": src, "padded": padded, "mask": mask, "dec": dec, "bad": bad, "blocks": blocks,
                "map": torch.empty_like(blocks), "radius": case["radius"]}
    reqs = []
    for w, h, kind, preset, s in _texture_list(case, seed, SERVE_MIX):
        img = _image(kind, w, h, s)
        mask = _outline(img).cpu().numpy() if kind == "alpha" else None
        reqs.append((img.cpu().numpy(), mask, _settings(preset)))
    return {"do": do, "reqs": reqs, "server": nb.Server(hbm_budget=1 << 30)}


def run(state):
    do = state["do"]
    if do == "cells":
        blocks = state["blocks"]
        blocks[:] = 0
        st = state["core"].compress(state["cells"], state["masks"], blocks)
        return {"blocks": blocks, "errs": [st.err_alpha, st.err_color], "ssim": [st.ssim_alpha, st.ssim_color]}
    if do == "device":
        dst = state["dst"]
        if state["start"] is None:
            dst.zero_()
        else:
            dst.copy_(state["start"])
        st = _encode(dst, state["bgra"], state["mask"], state["preset"], state["stats"])
        if st is None:
            return {"blocks": dst}
        return {"blocks": dst, "errs": [st.err_alpha, st.err_color], "ssim": [st.ssim_alpha, st.ssim_color]}
    if do == "image":
        enc = nb.encode_image(state["img"], state["flags"], state["preset"])
        st = enc.stats
        return {"blocks": enc.blocks, "errs": [st.err_alpha, st.err_color], "ssim": [st.ssim_alpha, st.ssim_color]}
    if do == "batch":
        state["batch"].launch(_stream())
        errs, ssim = state["batch"].sums(_stream())
        return {"blocks": [k[2] for k in state["keep"]], "errs": errs, "ssim": ssim}
    if do == "tools":
        lib, st = nb.load(), _stream()
        src, padded, mask, dec, bad, blocks = (state[k] for k in ("src", "padded", "mask", "dec", "bad", "blocks"))
        h, w = src.shape[:2]
        ph, pw = padded.shape[:2]
        check(lib.nebc7_prepare_device(src.data_ptr(), w * 4, w, h, padded.data_ptr(), mask.data_ptr(), state["radius"], st),
              "prepare")
        check(lib.nebc7_decode_device(blocks.data_ptr(), dec.data_ptr(), pw * 4, pw, ph, st), "decode")
        check(lib.nebc7_bad_blocks_device(padded.data_ptr(), dec.data_ptr(), mask.data_ptr(), pw * 4, pw, ph, 0, bad.data_ptr(),
                                          st), "bad")
        check(lib.nebc7_partition_map_device(blocks.data_ptr(), state["map"].data_ptr(), blocks.shape[0], st), "map")
        return {"padded": padded, "mask": mask, "decoded": dec, "bad": bad, "map": state["map"]}
    server = state["server"]
    outs, tickets = [], []
    for bgra, mask, settings in state["reqs"]:
        h, w = bgra.shape[:2]
        dst = np.zeros(((h // 4) * (w // 4), 16), np.uint8)
        outs.append(dst)
        tickets.append(server.submit(bgra, mask, dst, settings))
    errs = [server.wait(t)["errs"] for t in tickets]
    return {"blocks": outs, "errs": np.array(errs)}


def work(case):
    """Bytes: pixels, masks and starting blocks in, blocks (or the step's
    images) out, once each.  flops: the search's integer operations."""
    do = case["do"]
    if do == "tools":
        pw, ph = nb.padded_size(case["w"], case["h"])
        px, n = pw * ph, pw * ph // 16
        # source, padded and mask; blocks and decoded; the glitch map's three inputs and output; map in and out
        return {"bytes": case["w"] * case["h"] * 4 + 8 * px + 16 * n + 4 * px + 16 * px + 32 * n, "flops": 10 * px}
    if do in ("batch", "serve"):
        todo = [(w * h, kind == "alpha", preset) for w, h, kind, preset, _ in
                _texture_list(case, 0, BATCH_MIX if do == "batch" else SERVE_MIX)]
    elif do == "cells":
        todo = [(case["n"] * 16, True, case["preset"])]
    elif do == "image":
        pw, ph = nb.padded_size(case["w"], case["h"])
        preset = {"/draft": "draft", "/slow": "slow"}.get(case["flags"], "default" if case["denoise"] else "precise")
        todo = [(pw * ph, case["flags"] != "/nomask", preset)]
    else:
        todo = [(case["w"] * case["h"], case["mask"], case["preset"])]
    return {"bytes": sum(px * 4 * (2 if masked else 1) + px * 2 for px, masked, _ in todo),
            "flops": sum(px // 16 * OPS_PER_BLOCK[p] for px, _, p in todo)}


def exact(case, seed):
    """Blocks, maps and error sums are whole numbers, equal or wrong; the
    SSIM sums depend on the encoded blocks."""
    return None
