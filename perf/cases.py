"""What a user of the library has it do, as cases that can be timed and compared.

Ranges.  Sizes come from the repository's own workloads (a 321 x 481 image, the 1024^2 image as 16 patches of
256^2 + 5-px halo, uneven rectangles of 200-700 px, 256^2 training patches in minibatches of 16) and from the
smallest inputs that the entry points accept.  Images are seeded Voronoi mosaics with a ramp and noise, one cell per
about 4096 pixels.  Contexts are kept for the life of the program, one per configuration, as a program that
works through many images keeps them.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ucm-mpi-gpu_gb300"))

import gpb  # noqa: E402
from gpb import learned, synth  # noqa: E402

MODES = {"plain": gpb.EIG_LANCZOS, "warm": gpb.EIG_WARM, "block": gpb.EIG_BLOCK, "learned": gpb.EIG_LEARNED,
         "training": gpb.EIG_LEARNED}
MAX_BATCH_PX = 1_200_000   # the largest drawn batch; the largest listed one is about twice that
LEARNED_CONVS = [(16, 16, 0, 1), (16, 16, 0, 1), (16, 32, 1, 1), (32, 32, 1, 1), (32, 64, 2, 1), (64, 64, 2, 1),
                 (64, 64, 3, 1), (64, 64, 3, 1), (128, 64, 2, 1), (64, 64, 2, 1), (96, 32, 1, 1), (32, 32, 1, 1),
                 (48, 16, 0, 1), (16, 16, 0, 1), (16, 32, 0, 0)]  # cin, cout, level, ReLU


def listed():
    return [
        # one small region of interest, start to end: launches, host round trips and their latency
        {"name": "gpb_small_64x80", "op": "gpb", "mode": "warm", "compat": 0, "api": "host", "sizes": "64x80"},
        # one photograph with the library's default parameters (the plain cold-start Lanczos solver)
        {"name": "gpb_photo_321x481_plain", "op": "gpb", "mode": "plain", "compat": 0, "api": "host",
         "sizes": "321x481"},
        # the 1024^2 image in one batch of 16 halo'd patches, device to device: the ordinary production call
        {"name": "gpb_batch_16x266_warm", "op": "gpb", "mode": "warm", "compat": 0, "api": "device",
         "sizes": " ".join("%dx%d" % (261 if i in (0, 3) else 266, 261 if j in (0, 3) else 266)
                           for i in range(4) for j in range(4))},
        # uneven rectangles of a large image in one batch, behind the reference engine's own layout: the largest call
        {"name": "gpb_uneven_12_damascene", "op": "gpb", "mode": "warm", "compat": 1, "api": "host",
         "sizes": "613x587 202x699 431x350 377x521 640x233 297x412 555x688 219x265 483x301 350x213 698x633 382x476"},
        # texton and Lab labels of a thumbnail, without allocation, on the caller's stream
        {"name": "labels_96x131", "op": "labels", "h": 96, "w": 131},
        # the same entry point at the largest image that it takes
        {"name": "labels_1024x1024", "op": "labels", "h": 1024, "w": 1024},
        # the network's fields of an ordinary image's patches
        {"name": "net_forward_4x321x481", "op": "net_forward", "n": 4, "h": 321, "w": 481},
        # one minibatch of the network's training: loss and gradient
        {"name": "net_grad_16x256x256", "op": "net_grad", "n": 16, "h": 256, "w": 256},
        # the contour map's regions: one photograph, planes on the host, doubled grid out
        {"name": "ucm_photo_321x481", "op": "ucm", "n": 1, "h": 321, "w": 481, "double": True},
        # the pieces of a 1024^2 image in one call
        {"name": "ucm_pieces_16x256x256", "op": "ucm", "n": 16, "h": 256, "w": 256, "double": True},
        # the classifier's descriptors of a patch's superpixels
        {"name": "superpixels_266x266", "op": "superpixels", "h": 266, "w": 266, "labels": 300, "bin_step": 8,
         "textons": True},
        # whole-image planes from a batch's patches, blended over the halo
        {"name": "stitch_1024_blend", "op": "stitch", "h": 1024, "w": 1024, "rows": 4, "cols": 4, "halo": 5,
         "stitch": 2},
    ]


def _side(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["gpb", "gpb", "gpb", "gpb", "labels", "net_forward", "net_grad", "ucm", "superpixels", "stitch"])
    if op == "gpb":
        mode = rng.choice(["warm", "warm", "plain", "block", "learned"])
        most = MAX_BATCH_PX // 4 if mode == "plain" else MAX_BATCH_PX
        n, sizes, px = _side(rng, 1, 16), [], 0
        for _ in range(n):
            h, w = _side(rng, 32, 700), _side(rng, 32, 700)
            if px + h * w > most:
                break
            sizes.append("%dx%d" % (h, w))
            px += h * w
        return {"op": op, "mode": mode, "compat": rng.randrange(2), "api": rng.choice(["host", "device"]),
                "sizes": " ".join(sizes) or "97x113"}
    if op == "labels":
        return {"op": op, "h": _side(rng, 32, 1024), "w": _side(rng, 32, 1024)}
    if op in ("net_forward", "net_grad"):
        h, w = _side(rng, 48, 512), _side(rng, 48, 512)
        return {"op": op, "n": max(1, min(_side(rng, 1, 16), (1 << 20) // (h * w))), "h": h, "w": w}
    if op == "ucm":
        h, w = _side(rng, 32, 512), _side(rng, 32, 512)
        return {"op": op, "n": max(1, min(_side(rng, 1, 16), (1 << 20) // (h * w))), "h": h, "w": w,
                "double": rng.random() < 0.75}
    if op == "superpixels":
        return {"op": op, "h": _side(rng, 64, 320), "w": _side(rng, 64, 320), "labels": _side(rng, 20, 2000),
                "bin_step": rng.choice([1, 8, 8, 16]), "textons": rng.random() < 0.5}
    h, w = _side(rng, 192, 1024), _side(rng, 192, 1024)
    return {"op": "stitch", "h": h, "w": w, "rows": rng.randrange(1, 5), "cols": rng.randrange(1, 5),
            "halo": rng.randrange(0, 11), "stitch": rng.randrange(3)}


# ------------------------------------------------------------------ inputs
def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split()]


def _packed(h, w, seed, cells=None):
    """An h x w seeded image as packed uint32 (B<<16 | G<<8 | R) in an int32 device tensor."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    cells = cells or max(6, h * w // 4096)
    sites = torch.rand((cells, 2), generator=g, device="cuda") * torch.tensor([h, w], device="cuda")
    colours = torch.rand((cells, 3), generator=g, device="cuda") * 255
    xs = torch.arange(w, device="cuda", dtype=torch.float32)
    lab = torch.empty((h, w), dtype=torch.int64, device="cuda")
    for y0 in range(0, h, 64):
        ys = torch.arange(y0, min(h, y0 + 64), device="cuda", dtype=torch.float32)
        d = (ys[:, None, None] - sites[:, 0]) ** 2 + (xs[None, :, None] - sites[:, 1]) ** 2
        lab[y0:y0 + 64] = d.argmin(-1)
    img = colours[lab] + (40.0 * xs / max(w - 1, 1))[None, :, None]
    img = img + 8.0 * torch.randn((h, w, 3), generator=g, device="cuda")
    v = img.round().clamp(0, 255).to(torch.int32)
    return ((v[..., 0] << 16) | (v[..., 1] << 8) | v[..., 2]).contiguous()


def _host(t):
    return t.cpu().numpy().view(np.uint32)


_kept = {}


def _codebook():
    if "codebook" not in _kept:
        img = synth.voronoi_image(192, 192, 24, 8.0, synth.SEED_BASE)
        _kept["codebook"] = synth.make_codebook(img, synth.SEED_BASE, n_sample=2048)
    return _kept["codebook"]


def _weights(mode):
    """The shipped weights for a learned-start solve, the ones that training begins from for the network's own calls."""
    if ("weights", mode) not in _kept:
        _kept[("weights", mode)] = np.load(learned.WEIGHTS) if mode == "learned" else learned.init_params()
    return _kept[("weights", mode)]


def _new_context(mode, compat):
    ctx = gpb.Context(_codebook(), eig_mode=MODES[mode], compat=compat)
    if mode in ("learned", "training"):
        ctx.learned_set(_weights(mode))
    return ctx


def _context(mode="warm", compat=0):
    """The program's context for a configuration."""
    if (mode, compat) not in _kept:
        _kept[(mode, compat)] = _new_context(mode, compat)
    return _kept[(mode, compat)]


def _net_inputs(case, seed):
    """Per patch and pixel: mPb (sparse ridges in [0, 1]), affinity degree (1..81) and 9 orthonormal smooth fields."""
    n, h, w = case["n"], case["h"], case["w"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    mpb, deg, vs = [], [], []
    for _ in range(n):
        ridge = torch.zeros((h, w), device="cuda")
        fields = []
        for k in range(9):
            a = torch.rand(5, generator=g, device="cuda")
            arg = a[0] * 6.28 + (0.2 + a[1]) * 12 * ys / h + (a[2] - 0.5) * 24 * xs / w
            fields.append(torch.tanh(3 * torch.sin(arg)) + 0.1 * torch.cos(7 * a[3] + 5 * xs / w))
            ridge = torch.maximum(ridge, a[4] * (1 - (torch.sin(arg) * 6).abs()).clamp(min=0))
        ridge = ridge * (torch.rand((h, w), generator=g, device="cuda") > 0.1)
        mpb.append(ridge.reshape(-1))
        deg.append((1 + 80 * (1 - ridge) * (0.6 + 0.4 * torch.rand((h, w), generator=g, device="cuda"))).reshape(-1))
        q, _ = np.linalg.qr(torch.stack(fields, -1).reshape(-1, 9).double().cpu().numpy())
        vs.append(torch.from_numpy(q).float().cuda().reshape(-1))
    return torch.cat(mpb), torch.cat(deg), torch.cat(vs)


def _planes(h, w, seed):
    """8 orientation planes in [0, 1] as the contour stage leaves them: ridges along region borders over a low floor."""
    rng = np.random.default_rng(seed)
    fy, fx = np.fft.fftfreq(h)[:, None], np.fft.rfftfreq(w)[None, :]
    low = np.exp(-2 * (np.pi * 6.0) ** 2 * (fy ** 2 + fx ** 2))
    fine = np.exp(-2 * (np.pi * 1.5) ** 2 * (fy ** 2 + fx ** 2))

    def smooth(k):
        v = np.fft.irfft2(np.fft.rfft2(rng.standard_normal((h, w))) * k, s=(h, w))
        return v / v.std()
    ridge = np.exp(-np.abs(smooth(low)) * 4) + 0.5 * np.exp(-np.abs(smooth(low)) * 6)
    out = np.stack([0.05 + ridge * (0.6 + 0.4 * np.cos(2 * (smooth(low) - o * np.pi / 8))) + 0.03 * np.abs(smooth(fine))
                    for o in range(8)])
    return np.ascontiguousarray(((out - out.min()) / (out.max() - out.min())).astype(np.float32))


def _superpixel_inputs(case, seed):
    h, w, n = case["h"], case["w"], case["labels"]
    img = _packed(h, w, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    sites = torch.rand((n, 2), generator=g, device="cuda") * torch.tensor([h, w], device="cuda")
    ys = torch.arange(h, device="cuda", dtype=torch.float32)
    xs = torch.arange(w, device="cuda", dtype=torch.float32)
    lab = torch.stack([((ys[y] - sites[:, 0]) ** 2 + (xs[:, None] - sites[:, 1]) ** 2).argmin(-1) for y in range(h)])
    return img, lab.to(torch.int32).contiguous()


def prepare(case, seed):
    op = case["op"]
    if op == "gpb":
        ctx, sizes = _context(case["mode"], case["compat"]), _sizes(case)
        imgs = [_packed(h, w, seed * 1000 + i) for i, (h, w) in enumerate(sizes)]
        if case["api"] == "host":
            return {"op": op, "ctx": ctx, "packed": [_host(t) for t in imgs]}
        off = np.concatenate([[0], np.cumsum([h * w for h, w in sizes])])
        flat = torch.cat([t.reshape(-1) for t in imgs])
        n = int(off[-1])
        return {"op": "gpb_device", "ctx": ctx, "w": [s[1] for s in sizes], "h": [s[0] for s in sizes],
                "off": off[:-1], "packed": flat, "nmax": torch.empty(n, device="cuda"),
                "orient": torch.empty(8 * n, device="cuda")}
    if op == "labels":
        img = _packed(case["h"], case["w"], seed)
        return {"op": op, "ctx": _context(), "h": case["h"], "w": case["w"], "packed": img,
                "labels": torch.empty((case["h"], case["w"]), dtype=torch.int32, device="cuda")}
    if op in ("net_forward", "net_grad"):
        mpb, deg, v = _net_inputs(case, seed)
        st = {"op": op, "ctx": _context("training"), "shapes": [(case["h"], case["w"])] * case["n"], "mpb": mpb,
              "deg": deg}
        if op == "net_grad":
            st["v"] = v
        else:
            st["y"] = torch.empty((mpb.numel(), 32), device="cuda")
        return st
    if op == "ucm":
        return {"op": op, "ctx": _context(), "double": case["double"],
                "planes": [_planes(case["h"], case["w"], seed * 1000 + i) for i in range(case["n"])]}
    if op == "superpixels":
        img, lab = _superpixel_inputs(case, seed)
        ctx = _new_context("warm", 0)  # holds the patch's texton map and grey image
        ctx.compute_batch([_host(img)])
        cols = (32 if case["textons"] else 0) + 255 // case["bin_step"] + 1 + 4
        return {"op": op, "ctx": ctx, "labels": lab, "n": case["labels"], "bin_step": case["bin_step"],
                "textons": case["textons"],
                "out": torch.empty((case["labels"], cols), dtype=torch.float64, device="cuda")}
    h, w = case["h"], case["w"]
    img = _host(_packed(h, w, seed))
    boxes = synth.grid_patches(h, w, case["rows"], case["cols"], case["halo"])
    ctx = _new_context("warm", 0)  # holds the batch's planes
    ctx.compute_batch([np.ascontiguousarray(img[y:y + ph, x:x + pw]) for (y, x, ph, pw, *_r) in boxes])
    return {"op": "stitch", "ctx": ctx, "h": h, "w": w, "mode": case["stitch"], "ramp": max(1, case["halo"]),
            "places": [(x, y, ix, iy, iw, ih) for (y, x, ph, pw, iy, ix, ih, iw) in boxes],
            "nmax": torch.empty((h, w), device="cuda"), "orient": torch.empty((8, h, w), device="cuda")}


# -------------------------------------------------------------------- runs
def run(state):
    op, ctx = state["op"], state["ctx"]
    if op == "gpb":
        return ctx.compute_batch(state["packed"])
    if op == "gpb_device":
        ctx.compute_batch_device(state["w"], state["h"], state["off"], state["packed"].data_ptr(),
                                 state["nmax"].data_ptr(), state["orient"].data_ptr())
        return state["nmax"], state["orient"]
    if op == "labels":
        ctx.texton_labels_static(state["w"], state["h"], state["packed"].data_ptr(), state["labels"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream or 1)  # 1: the legacy default stream
        return state["labels"]
    if op == "net_forward":
        ctx.learned_forward_device(state["shapes"], state["mpb"].data_ptr(), state["deg"].data_ptr(),
                                   state["y"].data_ptr())
        return state["y"]
    if op == "net_grad":
        return ctx.learned_grad_device(state["shapes"], state["mpb"].data_ptr(), state["deg"].data_ptr(),
                                       state["v"].data_ptr())
    if op == "ucm":
        if len(state["planes"]) == 1:
            return ctx.ucm(state["planes"][0], double_size=state["double"])[0]
        return [m for m, _ in ctx.ucm_batch(state["planes"], double_size=state["double"])]
    if op == "superpixels":
        ctx.superpixel_features(0, state["labels"].data_ptr(), state["n"], state["out"].data_ptr(),
                                bin_step=state["bin_step"], with_textons=state["textons"])
        return state["out"]
    ctx.stitch_device(state["mode"], state["w"], state["h"], state["places"], state["nmax"].data_ptr(),
                      state["orient"].data_ptr(), ramp=state["ramp"])
    return state["nmax"], state["orient"]


# ------------------------------------------------------------------- exact
def _net_loss_and_fields(case, seed, grad):
    mpb, deg, v = _net_inputs(case, seed)
    n, h, w = case["n"], case["h"], case["w"]
    p = torch.from_numpy(_weights("training")).cuda().double().requires_grad_(grad)
    convs, at = [], 0
    for ci, co, _, _ in LEARNED_CONVS:
        wt = p[at:at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        at += co * 9 * ci
        convs.append((wt, p[at:at + co]))
        at += co
    x = torch.zeros((n, 16, h, w), dtype=torch.float64, device="cuda")
    x[:, 0], x[:, 1] = mpb.double().reshape(n, h, w), deg.double().reshape(n, h, w) / 81

    def conv(k, t):
        wt, b = convs[k]
        hh, ww = t.shape[2:]
        tp = torch.nn.functional.pad(t, (1, 1, 1, 1))
        z = b[None, :, None, None].expand(t.shape[0], -1, hh, ww)
        for dy in range(3):
            for dx in range(3):
                z = z + torch.einsum("oc,nchw->nohw", wt[:, :, dy, dx], tp[:, :, dy:dy + hh, dx:dx + ww])
        return torch.relu(z) if LEARNED_CONVS[k][3] else z

    def up(t, like):
        t = t.repeat_interleave(2, 2).repeat_interleave(2, 3)
        return t[:, :, :like.shape[2], :like.shape[3]]

    def pool(t):
        return torch.nn.functional.avg_pool2d(t, 2, ceil_mode=True, count_include_pad=False)
    s0 = conv(1, conv(0, x))
    s1 = conv(3, conv(2, pool(s0)))
    s2 = conv(5, conv(4, pool(s1)))
    t = conv(7, conv(6, pool(s2)))
    t = conv(9, conv(8, torch.cat([up(t, s2), s2], 1)))
    t = conv(11, conv(10, torch.cat([up(t, s1), s1], 1)))
    t = conv(13, conv(12, torch.cat([up(t, s0), s0], 1)))
    y = conv(14, t).permute(0, 2, 3, 1).reshape(n, h * w, 32)
    if not grad:
        return y.detach().reshape(-1, 32)
    vs = v.double().reshape(n, h * w, 9)
    gram = y.transpose(1, 2) @ y
    tr = gram.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None]
    gram = gram + 1e-4 * tr / 32 * torch.eye(32, dtype=torch.float64, device="cuda")
    b = vs.transpose(1, 2) @ y
    loss = (9 - (b @ torch.linalg.inv(gram) @ b.transpose(1, 2)).diagonal(dim1=1, dim2=2).sum(-1)).sum()
    loss.backward()
    return float(loss), p.grad.cpu().numpy()


def exact(case, seed):
    op = case["op"]
    if op == "net_forward":
        return _net_loss_and_fields(case, seed, False)
    if op == "net_grad":
        return _net_loss_and_fields(case, seed, True)
    if op == "superpixels" and not case["textons"]:
        img, lab = _superpixel_inputs(case, seed)
        v, lab, n = _host(img).astype(np.int64).ravel(), lab.cpu().numpy().ravel(), case["labels"]
        b, g, r = v >> 16, (v >> 8) & 255, v & 255
        grey = (r * 4899 + g * 9617 + b * 1868 + (1 << 13)) >> 14
        bins = 255 // case["bin_step"] + 1
        size = np.maximum(np.bincount(lab, minlength=n), 1).astype(np.float64)
        hist = np.bincount(lab * bins + grey // case["bin_step"], minlength=n * bins).reshape(n, bins)
        mean = np.stack([np.bincount(lab, weights=c, minlength=n) for c in (b, g, r)], 1)
        return np.concatenate([hist / size[:, None] * 10, np.zeros((n, 1)), mean / size[:, None] * (10 / 255)], 1)
    # labels are whole numbers; the contour stage's eigensolver, the contour map's greedy merge and the planes that
    # a stitch reads have no plain 64-bit form of a few seconds
    return None


# -------------------------------------------------------------------- work
def work(case):
    op = case["op"]
    if op == "gpb":
        px = sum(h * w for h, w in _sizes(case))
        # per pixel: 325 ring groups x 13 filters, half-disc counts of 4 cues, the 81-neighbour affinities, and one
        # degree-42 filter of a 32-vector block; the solver's repetitions are not counted
        return {"bytes": 40.0 * px, "flops": px * (2401 + 2.0 * 325 * 13 + 4 * 1257 + 81 * 10 + 42 * 81 * 32 * 2.0)}
    px = case["h"] * case["w"]
    if op == "labels":
        return {"bytes": 8.0 * px, "flops": px * (2401 + 2.0 * 325 * 13 + 3.0 * 13 * 32)}
    if op in ("net_forward", "net_grad"):
        px *= case["n"]
        flops = sum(2.0 * 9 * ci * co * px / 4 ** lv for ci, co, lv, _ in LEARNED_CONVS)
        if op == "net_forward":
            return {"bytes": px * (8.0 + 128), "flops": flops}
        return {"bytes": px * (8.0 + 36), "flops": 3 * flops}
    if op == "ucm":
        return {"bytes": case["n"] * px * (32.0 + (32.0 if case["double"] else 8.0)), "flops": 0.0}
    if op == "superpixels":
        cols = (32 if case["textons"] else 0) + 255 // case["bin_step"] + 1 + 4
        return {"bytes": px * 13.0 + 8.0 * cols * case["labels"], "flops": 0.0}
    inner = 36.0 * sum(ph * pw for (_, _, ph, pw, *_r) in
                       synth.grid_patches(case["h"], case["w"], case["rows"], case["cols"], case["halo"]))
    return {"bytes": inner + 36.0 * px, "flops": 0.0}
