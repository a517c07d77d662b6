"""The work that users of this framework have it do, as measurable cases: frame pairs interpolated at the sizes, formats
and multipliers of real sessions, motion blur, the mixed batch, the CNN-seeded estimate and the seed net's training.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what a program has in hand: frames on the GPU, the Interpolator / Batch / net it keeps
    run(state)            one pass through the public entry points; returns the generated frames (or loss and gradients)
    work(case)            bytes and operations of one pass: inputs read once, outputs written once, the method's arithmetic
    exact(case, seed)     the float64 value of what run returns, where it has one (the training pass)

Kinds of case:
    pair    one frame pair: the estimate, then m - 1 syntheses at t = k / m
    blur    one frame pair: the estimate, then one motion-blurred frame of n sub-frames
    batch   many pairs of mixed sizes, formats and multipliers recorded as one Batch
    train   one loss-and-gradient pass of the seed net on a batch of 256 x 256 crops (64 x 64 level-1 luma)
"""
import math
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "frame-gen-ritz_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import framegen as fg  # noqa: E402
import seednet_train  # noqa: E402
import workloads_gpu  # noqa: E402

# format name -> (view format, extra init arguments, bytes per pixel)
FORMATS = {
    "rgba8": (fg.VK_R8G8B8A8_UNORM, {}, 4.0),
    "bgra8": (fg.VK_B8G8R8A8_UNORM, {}, 4.0),
    "rgb10": (fg.VK_A2B10G10R10_UNORM, {}, 4.0),
    "f16lin": (fg.VK_R16G16B16A16_SFLOAT, {"transfer": 1}, 8.0),   # scRGB linear light, mismatch in PQ codes
    "f16enc": (fg.VK_R16G16B16A16_SFLOAT, {"transfer": 0}, 8.0),   # display encoded
    "nv12": (fg.VK_R8_UNORM, {"yuv_matrix": 1}, 1.5),
    "p010": (fg.VK_R16_UNORM, {"yuv_matrix": 2}, 3.0),
}


def _pair(name, fmt, w, h, mult, **more):
    return {"name": name, "kind": "pair", "fmt": fmt, "w": w, "h": h, "mult": mult, "fs": 2, "content": "flow", "ui": False,
            "cnn": False, **more}


def listed():
    return [
        # a small game window or emulator output doubled: the shortest chain of launches, latency counts
        _pair("rgba8_360p_x2", "rgba8", 640, 360, 2),
        # the ordinary case: a 1080p game doubled
        _pair("rgba8_1080p_x2", "rgba8", 1920, 1080, 2),
        # a laptop panel in BGRA order with tight (not 16-byte) rows, a protected crosshair, tripled; fresh content
        _pair("bgra8_768p_ui_x3", "bgra8", 1366, 768, 3, ui=True, content="fresh"),
        # a 4K game at 4x: the headline workload
        _pair("rgba8_4k_x4", "rgba8", 3840, 2160, 4),
        # the largest frames the library is used on
        _pair("rgba8_8k_x2", "rgba8", 7680, 4320, 2),
        # decoded SDR video doubled
        _pair("nv12_1080p_x2", "nv12", 1920, 1080, 2),
        # decoded HDR video doubled
        _pair("p010_4k_x2", "p010", 3840, 2160, 2),
        # a 4K HDR game in linear light, tripled
        _pair("f16lin_4k_x3", "f16lin", 3840, 2160, 3),
        # the 4K game with the CNN-seeded estimate
        _pair("rgba8_4k_cnn_x4", "rgba8", 3840, 2160, 4, cnn=True),
        # motion blur of a 4K game: 4 Gaussian samples over half a frame time
        {"name": "blur_4k_n4", "kind": "blur", "fmt": "rgba8", "w": 3840, "h": 2160, "n": 4, "fs": 2, "content": "flow"},
        # a server's batch: 16 pairs, 720p .. 2160p in ratio 9:4:2:1, four formats, 2x / 3x / 4x
        {"name": "batch_16_mixed", "kind": "batch", "slots": 16, "scale": 1.0},
        # a training step's loss and gradients on 64 crops
        {"name": "train_64", "kind": "train", "crops": 64, "crop": 256},
    ]


def _size(rng, lo, hi):
    """a frame size of lo .. hi pixels (spread over the logarithm), 4:3 .. 21:9, odd sizes among them"""
    area = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.choice((16 / 9, 16 / 9, 4 / 3, 16 / 10, 21 / 9))
    h = int(math.sqrt(area / aspect))
    w = int(h * aspect)
    if rng.random() < 0.5:   # an ordinary even size, else whatever came out
        w, h = w // 8 * 8, h // 2 * 2
    return max(w, 64), max(h, 64)


def draw(rng):
    r = rng.random()
    if r < 0.08:
        return {"kind": "train", "crops": rng.randint(4, 64), "crop": rng.choice((128, 256))}
    if r < 0.14:
        return {"kind": "batch", "slots": rng.randint(3, 16), "scale": rng.choice((0.25, 0.5, 0.75))}
    fmt = rng.choice(("rgba8", "rgba8", "rgba8", "bgra8", "rgb10", "f16lin", "f16enc", "nv12", "p010"))
    content = rng.choice(("flow", "flow", "flow", "fresh", "static"))
    fs = rng.choice((2, 2, 2, 2, 2, 1, 4))
    if r < 0.26:
        w, h = _size(rng, 320 * 180, 1920 * 1080)
        return {"kind": "blur", "fmt": fmt, "w": w, "h": h, "n": rng.randint(2, 6), "fs": fs, "content": content}
    w, h = _size(rng, 320 * 180, 3840 * 2160 if fs != 1 else 1920 * 1080)
    ui = fmt in ("rgba8", "bgra8") and rng.random() < 0.2
    cnn = fmt in ("rgba8", "bgra8") and not ui and fs == 2 and w * h > 1280 * 720 and rng.random() < 0.25
    return {"kind": "pair", "fmt": fmt, "w": w, "h": h, "mult": rng.randint(2, 4), "fs": fs, "content": content, "ui": ui,
            "cnn": cnn}


# ------------------------------------------------------------------------------------------------------- frames
def _encode(fmt, rgba):
    """an (H, W, 4) uint8 R,G,B,A frame as a frame of the format (YUV: a (Y, CbCr) tuple), limited-range codes"""
    if fmt == "rgba8":
        return rgba.contiguous()
    if fmt == "bgra8":
        return rgba[..., [2, 1, 0, 3]].contiguous()
    if fmt == "rgb10":
        v = rgba[..., :3].to(torch.int32)
        c = 4 * v + (v >> 6)
        return c[..., 0] | (c[..., 1] << 10) | (c[..., 2] << 20) | (-1 << 30)
    e = rgba[..., :3].float() / 255.0
    if fmt in ("f16lin", "f16enc"):
        rgb = torch.pow(10.0, -3.0 + 4.0 * e) if fmt == "f16lin" else e
        return torch.cat([rgb, torch.ones_like(rgb[..., :1])], dim=-1).to(torch.float16).contiguous()
    kr, kb = (0.2126, 0.0722) if fmt == "nv12" else (0.2627, 0.0593)
    q = 1 if fmt == "nv12" else 4
    y = kr * e[..., 0] + (1 - kr - kb) * e[..., 1] + kb * e[..., 2]
    c = torch.stack([(e[..., 2] - y) / (2 * (1 - kb)), (e[..., 0] - y) / (2 * (1 - kr))])
    H, W = y.shape
    c = torch.nn.functional.pad(c[None], (0, W & 1, 0, H & 1), mode="replicate")
    c = torch.nn.functional.avg_pool2d(c, 2)[0]
    yc = torch.round(16 * q + 219 * q * y).to(torch.int32)
    cc = torch.round(128 * q + 224 * q * c).to(torch.int32).permute(1, 2, 0).contiguous()
    if fmt == "nv12":
        return yc.to(torch.uint8), cc.to(torch.uint8)
    return (yc << 6).to(torch.int16), (cc << 6).to(torch.int16)


def _like(f):
    return tuple(torch.zeros_like(x) for x in f) if isinstance(f, tuple) else torch.zeros_like(f)


def _crosshair(f):
    """a static plus in the middle of the frame, as a game's overlay draws it"""
    H, W = f.shape[:2]
    y, x = H // 2, W // 2
    f[y - 1:y + 1, x - 6:x + 6, :3] = torch.tensor([0, 255, 0], dtype=torch.uint8, device=f.device)
    f[y - 6:y + 6, x - 1:x + 1, :3] = torch.tensor([0, 255, 0], dtype=torch.uint8, device=f.device)


def _frames(case, gen):
    """(prev, curr) of the case's format and size: smooth motion of up to 24 px; content "fresh": a fifth of the frame
    is new in curr; "static": nothing moves. Linear F16: a pan with rigid sprites, log-uniform light."""
    w, h, fmt, content = case["w"], case["h"], case["fmt"], case["content"]
    if fmt == "f16lin" and content == "flow":
        s = min(w, h)
        return workloads_gpu.hdr_pair(w, h, gen, smin=max(8, s // 17), smax=max(16, s // 6))
    d = workloads_gpu.flow_batch(1, w, h, gen, cut_frac=0.0, fresh_frac=1.0 if content == "fresh" else 0.0)
    p = d["prev"][0]
    c = p.clone() if content == "static" else d["curr"][0]
    if case.get("ui"):
        _crosshair(p)
        _crosshair(c)
    return _encode(fmt, p), _encode(fmt, c)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


# ------------------------------------------------------------------------------------------------------- state
def _interpolator(case, settings):
    vk, extra, _ = FORMATS[case["fmt"]]
    it = fg.Interpolator()
    if not it.init(case["w"], case["h"], vk, settings=settings, **extra):
        raise RuntimeError(it.init_error())
    return it


def _slots(case):
    """the batch's (w, h, fmt, multiplier): sizes in ratio 9:4:2:1 from the largest down, formats and multipliers cycling"""
    sizes = ([(3840, 2160)] + [(2560, 1440)] * 2 + [(1920, 1080)] * 4 + [(1280, 720)] * 9)[16 - case["slots"]:]
    fmts = ("p010", "rgb10", "rgba8", "nv12")
    return [(max(64, int(w * case["scale"])), max(64, int(h * case["scale"])), fmts[i % 4], 2 + i % 3)
            for i, (w, h) in enumerate(sizes)]


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "train":
        B, s = case["crops"], case["crop"]
        d = workloads_gpu.flow_batch(B, s, s, gen, cut_frac=0.0, fresh_frac=0.0)

        def luma(f):   # level 1 at flowScale 2: the mean luma of 4 x 4 pixels
            y = f[..., 0].float() * 0.299 + f[..., 1].float() * 0.587 + f[..., 2].float() * 0.114
            return torch.nn.functional.avg_pool2d(y[:, None], 4)[:, 0].contiguous()

        x = fg.SeedNet.pack(luma(d["prev"]), luma(d["curr"]))
        bs = s // 4 // 8
        truth = d["v"].reshape(B, bs, s // bs, bs, s // bs, 2).mean(dim=(2, 4)) / 8.0
        tgt = torch.zeros(B, bs, bs, 6, device="cuda")
        tgt[..., 0:2] = truth
        tgt[..., 2:4] = torch.round(truth)   # the plain search's integer vectors
        tgt[..., 4] = 1.0
        net = fg.SeedNet(B, s // 4, s // 4)
        params = seednet_train.init_params(seed)
        net.set_params(params)
        grad = net.grad_buffer()
        grad.net = net   # the view is valid while its net lives: whoever holds the view holds the net
        return {"kind": kind, "net": net, "grad": grad, "x": x, "tgt": tgt, "params": params,
                "loss": torch.zeros(1, dtype=torch.float32, device="cuda")}
    if kind == "batch":
        b = fg.Batch()
        prev, curr, outs = [], [], []
        for i, (w, h, fmt, m) in enumerate(_slots(case)):
            vk, extra, _ = FORMATS[fmt]
            if b.add(w, h, vk, multiplier=m, **extra) != i:
                raise RuntimeError(b.error())
            p, c = _frames({"w": w, "h": h, "fmt": fmt, "content": "flow"}, gen)
            prev.append(p)
            curr.append(c)
            outs += [_like(p) for _ in range(m - 1)]
        return {"kind": kind, "batch": b, "prev": prev, "curr": curr, "outs": outs}
    prev, curr = _frames(case, gen)
    if kind == "blur":
        it = _interpolator(case, fg.Settings(blurSamples=case["n"], flowScale=case["fs"]))
        return {"kind": kind, "it": it, "prev": prev, "curr": curr, "outs": [_like(prev)]}
    settings = fg.Settings(flowScale=case["fs"])
    if case["ui"]:
        settings.uiProtection, settings.uiEstimateFill = 3, True
    it = _interpolator(case, settings)
    if case["cnn"]:
        params = np.fromfile(os.path.join(PKG, "seednet_l1.bin"), np.float32)
        if not it.set_seed_net(params, 1):
            raise RuntimeError(it.last_error())
    if case["ui"]:   # the session has been running: the crosshair has been seen in the frames before this pair
        for k in range(10):
            it.begin_frame()
            if not it.record_observe(curr if k & 1 else prev):
                raise RuntimeError(it.last_error())
    m = case["mult"]
    return {"kind": kind, "it": it, "prev": prev, "curr": curr, "ui": case["ui"],
            "times": [float(np.float32(k) / np.float32(m)) for k in range(1, m)], "outs": [_like(prev) for _ in range(m - 1)]}


def run(state):
    kind = state["kind"]
    if kind == "train":   # the gradients of one step (the Adam update is left out: the same pass can be taken again)
        net = state["net"]
        net.zero_grads()
        net.backward(state["x"], state["tgt"], state["loss"])
        return {"loss": state["loss"], "grad": state["grad"]}
    if kind == "batch":
        if not state["batch"].record(state["prev"], state["curr"], state["outs"]):
            raise RuntimeError(state["batch"].error())
        return state["outs"]
    it, prev, curr = state["it"], state["prev"], state["curr"]
    it.begin_frame()
    if kind == "blur":
        if not it.record_estimate(prev, curr) or not it.record_synth_blur(prev, curr, state["outs"][0], 0.25, 0.75):
            raise RuntimeError(it.last_error())
        return state["outs"]
    if state["ui"] and not it.record_observe(curr):
        raise RuntimeError(it.last_error())
    if not it.record_estimate(prev, curr):
        raise RuntimeError(it.last_error())
    for out, t in zip(state["outs"], state["times"]):
        if not it.record_synth(prev, curr, out, t):
            raise RuntimeError(it.last_error())
    return state["outs"]


# ------------------------------------------------------------------------------------------------------- work
def _estimate_flops(w, h, fs):
    """the estimate's arithmetic per flow pixel: 25 integer candidates and 6 seeds scored by |a - c| sums (3 each), over
    all levels (4/3); 18 sub-pixel candidates (two bilinear taps and the sum, 17 each); 6 candidate vectors' errors
    (two taps, |a - c| and a separable 5 x 5 box, 21 each)"""
    return (w / fs) * (h / fs) * (31 * 3 * 4 / 3 + 18 * 17 + 6 * 21)


def _synth_flops(w, h):
    """a synthesis' arithmetic per pixel: the half-vector (12), two 3-channel bilinear warps (42), the largest channel
    difference (6), a separable 7 x 7 box (4), the trust ramp and the blend (14)"""
    return w * h * 78.0


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["crops"]
        s = case["crop"] // 4
        macs = 0.0
        for ci, co, st in zip((2, 32, 32, 32, 32, 32), (32, 32, 32, 32, 32, 8), (2, 2, 2, 1, 1, 1)):
            s = (s + st - 1) // st
            macs += n * s * s * 9.0 * ci * co
        x = n * (case["crop"] // 4) ** 2 * 4.0 + n * s * s * 24.0
        return {"bytes": x + 39912 * 8.0, "flops": 6.0 * macs}
    if kind == "batch":
        b = f = 0.0
        for w, h, fmt, m in _slots(case):
            b += (m + 1) * w * h * FORMATS[fmt][2]
            f += _estimate_flops(w, h, 2) + (m - 1) * _synth_flops(w, h)
        return {"bytes": b, "flops": f}
    w, h, px = case["w"], case["h"], FORMATS[case["fmt"]][2]
    synths, outs = (case["n"], 1) if kind == "blur" else (case["mult"] - 1, case["mult"] - 1)
    return {"bytes": (2 + outs) * w * h * px, "flops": _estimate_flops(w, h, case["fs"]) + synths * _synth_flops(w, h)}


# ------------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    """Generated frames are codes chosen by discrete decisions (search minima, roundings of positions to 1/32 px) and
    have no float64 value of their own: None. The training pass: the net, the loss and its gradients in float64."""
    if case["kind"] != "train":
        return None
    st = prepare(case, seed)
    p = torch.from_numpy(st["params"]).cuda().double()
    layers, o = [], 0
    for ci, co in zip((2, 32, 32, 32, 32, 32), (32, 32, 32, 32, 32, 8)):
        w = p[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
        b = p[o + co * 9 * ci:o + co * (9 * ci + 1)].clone().requires_grad_(True)
        layers.append((w, b))
        o += co * (9 * ci + 1)
    h = st["x"].double().permute(0, 3, 1, 2)
    for i, (w, b) in enumerate(layers):
        h = torch.nn.functional.conv2d(h, w, b, stride=2 if i < 3 else 1, padding=1)
        if i < 5:
            h = torch.relu(h)
    out, t = h.permute(0, 2, 3, 1), st["tgt"].double()
    e = out[..., :4] - t[..., :4]
    ae = e.abs()
    hub = torch.where(ae < 1, 0.5 * e * e, ae - 0.5).sum(-1)
    y = (ae[..., :2].amax(-1) < 1).double()
    z = out[..., 4]
    bce = torch.clamp(z, min=0) - z * y + torch.log1p(torch.exp(-z.abs()))
    loss = (t[..., 4] * (hub + bce)).mean()
    loss.backward()
    grad = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad]) for w, b in layers])
    return {"loss": loss.detach().reshape(1), "grad": grad}
