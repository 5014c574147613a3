"""The work a user has this framework do, as cases to be timed through its
public entry points: edge detection of single images, of batches and of
batches held in host memory, the two direction extensions, the training step
with its backward pass, and the subpixel third-order correction of dense edge
maps.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call, ``run`` is one call, ``work`` what the call cannot do without
and ``exact`` its result in 64 bits from plain torch.
"""
import importlib.util
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = "cuda:0"
EDGEL_SHARE = 0.03  # edgels per pixel of the generated images, about


def _package():
    """The package (its folder's name is no Python identifier)."""
    name = "toed_gb300"
    if name not in sys.modules:
        folder = os.path.join(ROOT, "third-order-edge-detector_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one thumbnail or crop, its count read back at once
        _detect("crop_97x150_u8", n=1, h=97, w=150, dtype="u8", sigma=2.0, how="call"),
        # the reference's own use: one camera frame in, the edgel list out (752 x 480, 8 bit)
        _detect("frame_480x752_u8", n=1, h=480, w=752, dtype="u8", sigma=1.0, how="call"),
        # one HD frame of the precision study, its list awaited
        _detect("frame_1080x1920_f32", n=1, h=1080, w=1920, dtype="f32", sigma=2.0, how="call"),
        # a 4K video stream: frames detected one after another into kept buffers
        _detect("stream_2160x3840_f32", n=1, h=2160, w=3840, dtype="f32", sigma=1.0, how="into"),
        # the uneven batch of 64 images, replayed from a CUDA graph
        _detect("batch_uneven64_f32", n=64, lo=256, hi=2048, dtype="f32", sigma=1.5, how="graph"),
        # a folder of 8-bit photographs of odd sizes, positions wanted in FP64
        _detect("batch_odd12_u8_f64", n=12, lo=301, hi=1501, dtype="u8", sigma=2.0, how="into", out="f64"),
        # the uneven batch in host memory: images in, lists out
        _detect("host_uneven64_f32", n=64, lo=256, hi=2048, dtype="f32", sigma=1.5, how="host"),
        # the MATLAB quick-and-dirty orientation on a batch
        _detect("qad_uneven8_f32", n=8, lo=256, hi=2048, dtype="f32", sigma=1.5, how="call", mode="qad"),
        # a training step: detection, loss on strength and position, gradients of pixels and sigma
        {"name": "train_16x512", "kind": "train", "n": 16, "h": 512, "w": 512, "sigma": 1.5},
        # the adjoint alone, gradients of all four edgel values given, odd image sizes
        {"name": "adjoint_6x777x1001", "kind": "adjoint", "n": 6, "h": 777, "w": 1001, "sigma": 2.0},
        # correction of a batch of learned edge-probability maps
        _maps("maps_8x2048", n=8, h=2048, w=2048, dtype="f32", sigma=2.0),
        # small double-precision maps with their own orientation, on the doubled work grid
        _maps("maps_2x251x334_f64", n=2, h=251, w=334, dtype="f64", sigma=1.5, theta=True, interp_n=1),
    ]


def _detect(name, n, dtype, sigma, how, h=0, w=0, lo=0, hi=0, out="f32", mode="grid", threshold=2.0):
    return {"name": name, "kind": "detect", "n": n, "h": h, "w": w, "lo": lo, "hi": hi, "dtype": dtype, "sigma": sigma,
            "how": how, "out": out, "mode": mode, "threshold": threshold}


def _maps(name, n, h, w, dtype, sigma, theta=False, interp_n=0):
    return {"name": name, "kind": "maps", "n": n, "h": h, "w": w, "dtype": dtype, "sigma": sigma, "theta": theta,
            "interp_n": interp_n, "thresh": 0.1, "radius": 2.0}


def draw(rng):
    """One more case of the same ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["single", "single", "batch", "batch", "host", "mode", "train", "adjoint", "maps", "maps"])
    sigma = rng.choice([0.7, 1.0, 1.5, 1.5, 2.0, 2.0, 2.5])
    if kind == "single":
        c = _detect("", 1, rng.choice(["u8", "f32"]), sigma, rng.choice(["call", "into"]), h=size(48, 2160),
                    w=size(48, 3840), out=rng.choice(["f32", "f32", "f64"]))
    elif kind == "batch":
        lo = size(64, 700)
        c = _detect("", rng.randint(2, 40), rng.choice(["u8", "f32"]), sigma, rng.choice(["into", "graph"]), lo=lo,
                    hi=min(2048, lo * rng.randint(2, 5)), out=rng.choice(["f32", "f32", "f64"]))
    elif kind == "host":
        lo = size(64, 700)
        c = _detect("", rng.randint(2, 24), rng.choice(["u8", "f32"]), sigma, "host", lo=lo,
                    hi=min(2048, lo * rng.randint(2, 5)))
    elif kind == "mode":
        lo = size(64, 600)
        c = _detect("", rng.randint(1, 8), rng.choice(["u8", "f32"]), rng.choice([1.0, 1.5, 2.0]), "call", lo=lo,
                    hi=lo * 3, mode=rng.choice(["qad", "qad", "normal", "fp32"]))
    elif kind == "train":
        c = {"kind": "train", "n": rng.randint(1, 16), "h": size(64, 700), "w": size(64, 700),
             "sigma": rng.choice([1.0, 1.5, 2.0])}
    elif kind == "adjoint":
        c = {"kind": "adjoint", "n": rng.randint(1, 8), "h": size(64, 1000), "w": size(64, 1000),
             "sigma": rng.choice([1.0, 1.5, 2.0])}
    else:
        fine = rng.random() < 0.25
        top = 500 if fine else 2048
        c = _maps("", rng.randint(1, 3 if fine else 8), size(64, top), size(64, top), rng.choice(["f32", "f32", "f64"]),
                  rng.choice([1.0, 1.5, 2.0, 2.0]), theta=rng.random() < 0.3, interp_n=1 if fine else 0)
    c.pop("name", None)
    c["sizes"] = rng.randrange(1 << 20)  # the seed of an uneven batch's sizes
    return c


def _sizes(case):
    """(H, W) of each image of a case: the same for every seed."""
    if not case.get("lo"):
        return [(case["h"], case["w"])] * case["n"]
    r = random.Random(case.get("sizes", 3000))
    lo, hi = case["lo"], case["hi"]
    step = 4 if lo % 2 == 0 else 1  # the uneven batch has multiples of 4, the odd folder any size
    return [tuple(max(lo, int(round(r.uniform(lo, hi) / step)) * step) for _ in range(2)) for _ in range(case["n"])]


# ---------------------------------------------------------------------------
# inputs: filled ellipses and convex polygons on 128, blurred, noisy; ridges
# ---------------------------------------------------------------------------
def _blur(img):
    x = torch.arange(-4, 5, dtype=torch.float32, device=DEV)
    k = torch.exp(-x * x / 2)
    k = k / k.sum()
    p = torch.nn.functional.pad(img[None, None], (4, 4, 4, 4), mode="reflect")[0, 0]
    h, w = img.shape
    rows = sum(k[t] * p[:, t:t + w] for t in range(9))
    return sum(k[t] * rows[t:t + h] for t in range(9))


def _shapes(h, w, gen, rng, noise, disc=False):
    """One float32 image in [0, 255]; with ``disc`` the last shape is the disc
    of radius min(h, w) / 4 around the image's centre."""
    img = torch.full((h, w), 128.0, device=DEV)
    scale = w / 752.0
    for _ in range(max(6, round(20 * h * w / (480 * 752)))):
        cx, cy, value = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(30, 220)
        radius = rng.uniform(10, 120) * scale
        if rng.random() < 0.5:
            corners, other, turn = None, rng.uniform(10, 120) * scale, rng.uniform(0, math.pi)
        else:
            corners = sorted(rng.uniform(0, 2 * math.pi) for _ in range(rng.randint(3, 8)))
            other = radius
        reach = max(radius, other) + 1
        x0, x1 = max(0, int(cx - reach)), min(w, int(cx + reach) + 2)
        y0, y1 = max(0, int(cy - reach)), min(h, int(cy + reach) + 2)
        if x0 >= x1 or y0 >= y1:
            continue
        dx = torch.arange(x0, x1, device=DEV, dtype=torch.float32)[None, :] - cx
        dy = torch.arange(y0, y1, device=DEV, dtype=torch.float32)[:, None] - cy
        if corners is None:
            c, s = math.cos(turn), math.sin(turn)
            inside = ((dx * c + dy * s) / radius) ** 2 + ((dy * c - dx * s) / other) ** 2 <= 1
        else:
            inside = torch.ones((y1 - y0, x1 - x0), dtype=torch.bool, device=DEV)
            for t, a in enumerate(corners):
                b = corners[(t + 1) % len(corners)]
                ax, ay, bx, by = (radius * f(v) for v in (a, b) for f in (math.cos, math.sin))
                inside &= (bx - ax) * (dy - ay) >= (by - ay) * (dx - ax)
        img[y0:y1, x0:x1].masked_fill_(inside, value)
    if disc:
        dx = torch.arange(w, device=DEV, dtype=torch.float32)[None, :] - w / 2
        dy = torch.arange(h, device=DEV, dtype=torch.float32)[:, None] - h / 2
        img.masked_fill_(dx * dx + dy * dy <= (min(h, w) / 4) ** 2, 200.0)
    img = _blur(img)
    return (img + noise * torch.randn((h, w), generator=gen, device=DEV)).clamp_(0, 255)


def _images(case, seed, disc=False):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rng = random.Random(seed)
    noise = 8 if case["sigma"] >= 1.5 else 3  # a narrow filter is for clean images
    out = []
    for h, w in _sizes(case):
        img = _shapes(h, w, gen, rng, rng.uniform(1, noise) if case["n"] > 1 else 3.0, disc)
        out.append(img.round().to(torch.uint8) if case.get("dtype") == "u8" else img)
    return out


def _ridges(h, w, gen, rng):
    """Edge-probability map: 40 cubic Bezier curves as Gaussian ridges of
    width 1.5 and peak U[0.5, 1], uniform noise to 0.05, clipped to [0, 1]."""
    E = torch.zeros(h * w, device=DEV)
    near = torch.arange(-5, 7, device=DEV)
    for _ in range(40):
        p = [(rng.uniform(0, w), rng.uniform(0, h)) for _ in range(4)]
        peak = rng.uniform(0.5, 1.0)
        length = sum(math.dist(p[i], p[i + 1]) for i in range(3))
        t = torch.linspace(0, 1, max(8, int(2 * length)), device=DEV)
        u = 1 - t
        x, y = (u ** 3 * a[0] + 3 * u * u * t * a[1] + 3 * u * t * t * a[2] + t ** 3 * a[3]
                for a in ([q[0] for q in p], [q[1] for q in p]))
        xs, ys = x.floor().long()[:, None] + near, y.floor().long()[:, None] + near
        gx, gy = torch.exp(-(xs - x[:, None]) ** 2 / 4.5), torch.exp(-(ys - y[:, None]) ** 2 / 4.5)
        value = peak * gy[:, :, None] * gx[:, None, :]
        value = value * ((ys >= 0) & (ys < h))[:, :, None] * ((xs >= 0) & (xs < w))[:, None, :]
        at = ys.clamp(0, h - 1)[:, :, None] * w + xs.clamp(0, w - 1)[:, None, :]
        E.scatter_reduce_(0, at.reshape(-1), value.reshape(-1), "amax")
    E = E.reshape(h, w) + 0.05 * torch.rand((h, w), generator=gen, device=DEV)
    return E.clamp_(0, 1)


def _ridge_maps(case, seed):
    """The maps and, where the case gives orientations, theirs: the tangent of
    the smoothed map's gradient."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rng = random.Random(seed)
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    maps = [_ridges(case["h"], case["w"], gen, rng).to(dt) for _ in range(case["n"])]
    if not case["theta"]:
        return maps, None
    thetas = []
    for E in maps:
        gy, gx = torch.gradient(_blur(E.float()))
        thetas.append(torch.remainder(torch.atan2(gy, gx), math.pi).to(dt).contiguous())
    return maps, thetas


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------
def _params(T, case):
    mode = case["mode"]
    return T.make_params(case["sigma"], 0, case["threshold"], 10, T.TOED_F64 if case["out"] == "f64" else T.TOED_F32,
                         T.TOED_FP32 if mode == "fp32" else T.TOED_HYBRID,
                         T.TOED_ORI_QAD if mode == "qad" else T.TOED_ORI_GRID,
                         T.TOED_NMS_TO_NORMAL if mode == "normal" else T.TOED_NMS_GRADIENT)


def _capacity(h, w):
    return h * w // 2


def _buffers(shapes, out, device):
    """One list, index and count buffer for a batch, and each image's part of them."""
    caps = [_capacity(h, w) for h, w in shapes]
    total, pin = sum(caps), device == "cpu"
    dt = torch.float64 if out == "f64" else torch.float32
    edgels = torch.zeros((total, 4), dtype=dt, device=device, pin_memory=pin)
    counts = torch.zeros(len(caps), dtype=torch.int32, device=device, pin_memory=pin)
    # a host program takes the lists alone
    index = None if pin else torch.zeros(total, dtype=torch.int32, device=device)
    outs, at = [], 0
    for k, cap in enumerate(caps):
        outs.append({"edgels": edgels[at:at + cap], "index": None if pin else index[at:at + cap],
                     "count": counts[k:k + 1], "capacity": cap})
        at += cap
    return outs, {"edgels": edgels, "index": index, "counts": counts}


def _edgel_grads(index, edgels):
    """dL/d(edgels) of some loss on the clear edges (a faint edgel's orientation
    means little), a function of the grid point."""
    i = index.to(torch.float64)
    return torch.stack([torch.cos(0.37 * i + k) for k in range(4)], 1) * (edgels[:, 3:] > 10)


def prepare(case, seed):
    T = _package()
    det = T.Detector(0)
    s = {"case": case, "T": T, "det": det}
    if case["kind"] == "detect":
        s["params"] = p = _params(T, case)
        images = _images(case, seed)
        shapes = [tuple(im.shape) for im in images]
        if case["how"] == "host":
            s["images"] = [im.cpu().pin_memory() for im in images]
            outs, s["buffers"] = _buffers(shapes, case["out"], "cpu")
            s["batch"] = det.host_batch(s["images"], outs)
        else:
            s["images"] = images
            s["outs"], s["buffers"] = _buffers(shapes, case["out"], DEV)
            s["lists"] = {k: [o[k] for o in s["outs"]] for k in ("edgels", "index")}
            if case["how"] == "graph":
                s["graph"] = det.capture(images, s["outs"], p)
    elif case["kind"] == "maps":
        s["maps"], s["thetas"] = _ridge_maps(case, seed)
        rows = (case["h"] << case["interp_n"]) * (case["w"] << case["interp_n"]) // 4
        s["lists"] = [torch.zeros((rows, 4), device=DEV) for _ in s["maps"]]
    else:
        s["images"] = torch.stack(_images(case, seed, disc=True))
        if case["kind"] == "train":
            s["images"].requires_grad_(True)
            s["sigma"] = torch.tensor(case["sigma"], device=DEV, requires_grad=True)
        else:
            s["images"] = list(s["images"])
            res = det.detect_batch(s["images"], sigma=case["sigma"])
            s["index"] = [r["index"].clone() for r in res]
            s["grads"] = [_edgel_grads(r["index"], r["edgels"]).float() for r in res]
    return s


def _train_loss(edgels, h, w):
    """(strength - 10)^2 plus the squared distance to the central disc's
    boundary, capped where the edgel is another shape's."""
    x, y, strength = edgels[:, 0] + 0.5, edgels[:, 1] + 0.5, edgels[:, 3]
    off = torch.sqrt((x - w / 2) ** 2 + (y - h / 2) ** 2) - min(h, w) / 4
    return ((strength - 10) ** 2).sum() + (off ** 2).clamp(max=9.0).sum()


def run(state):
    case, T, det = state["case"], state["T"], state["det"]
    if case["kind"] == "detect":
        p, how = state["params"], case["how"]
        if how == "graph":
            state["graph"].replay()
        elif how == "host":
            det.detect_host(state["batch"], params=p)
        else:
            det.detect_into(state["images"], state["outs"], p)
        if how == "call":  # the program goes on with the lists: how long are they?
            return {**state["lists"], "counts": state["buffers"]["counts"].tolist()}
        return state["buffers"]
    if case["kind"] == "maps":
        res = det.subpix_to_correct_batch(state["maps"], thresh=case["thresh"], sigma=case["sigma"],
                                          nbr_radius=case["radius"], thetas=state["thetas"], interp_n=case["interp_n"])
        for r, kept in zip(res, state["lists"]):
            kept[:r["count"]] = r["edgels"]
        return {"edgels": state["lists"], "counts": [r["count"] for r in res], "TO_E": [r["TO_E"] for r in res],
                "TO_O": [r["TO_O"] for r in res]}
    if case["kind"] == "train":
        images, sigma = state["images"], state["sigma"]
        edgels, counts, index = T.differentiable_detect(images, sigma, detector=det)
        loss = _train_loss(edgels, case["h"], case["w"])
        gi, gs = torch.autograd.grad(loss, [images, sigma])
        return {"loss": loss.detach(), "counts": counts, "grad_images": gi, "grad_sigma": gs}
    grads, gs = det.backward_batch(state["images"], state["index"], state["grads"], sigma=case["sigma"])
    return {"grad_images": grads, "grad_sigma": gs.float()}  # sigma is a float32 parameter


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    """Each input read once, each output written once; the separable form of
    the dense filters (the first derivatives and what feeds them, 64 r + 88
    operations a pixel) and the per-edgel sums at the edgels alone."""
    px = float(sum(h * w for h, w in _sizes(case)))
    r = math.ceil(4 * case["sigma"])
    n = EDGEL_SHARE * px
    if case["kind"] == "maps":
        fine = px * 4 ** case["interp_n"]
        esz = 8 if case["dtype"] == "f64" else 4
        return {"bytes": px * (esz * (2 if case["theta"] else 1) + 8) + 0.01 * px * 16,
                "flops": fine * (20 if case["theta"] else 70) + 0.01 * fine * (6 * 4 + 8) * 2 * (2 * r + 1)}
    detect = px * (64 * r + 88) + n * 14 * (2 * r + 3)
    adjoint = n * ((2 * r + 5) ** 2 * 12 + (2 * r + 5) * 100)
    if case["kind"] == "adjoint":
        return {"bytes": px * 8 + n * 20, "flops": adjoint}
    if case["kind"] == "train":
        return {"bytes": px * 12 + n * 40, "flops": detect + adjoint}
    point = n * (2 * r + 5) * (4 * 8 + 40) if case["mode"] == "qad" else 0.0
    return {"bytes": px * (1 if case["dtype"] == "u8" else 4)
            + n * ((32 if case["out"] == "f64" else 16) + (0 if case["how"] == "host" else 4)), "flops": detect + point}


# ---------------------------------------------------------------------------
# exact: the same results in 64 bits
# ---------------------------------------------------------------------------
def _taps64(sigma, r):
    """G, Gx, Gxx, Gxxx at whole offsets -(r+1)..r+1, then at offsets + 1/2; sigma a 0-d tensor."""
    x0 = torch.arange(-(r + 1), r + 2, dtype=torch.float64, device=DEV)
    rows, c, s = [], math.sqrt(2 * math.pi), sigma
    for shift in (0.0, 0.5):
        x = x0 + shift
        e = torch.exp(-x * x / (2 * s * s)) / c
        rows += [e / s, -x * e / s ** 3, (x * x - s * s) * e / s ** 5, x * (3 * s * s - x * x) * e / s ** 7]
    return torch.stack(rows)


#: the nine derivatives as (x filter, y filter): fx fy fxx fxy fyy fxxy fxyy fxxx fyyy
_NINE = [(1, 0), (0, 1), (2, 0), (1, 1), (0, 2), (2, 1), (1, 2), (3, 0), (0, 3)]


def _dense9(img, taps, r):
    """The nine derivatives on the half-pixel grid, (9, 2H, 2W), zero padding."""
    h, w = img.shape
    out = torch.empty((9, 2 * h, 2 * w), dtype=torch.float64, device=DEV)
    p = torch.nn.functional.pad(img, (r + 1,) * 4)

    def conv(a, t, dim, size, whole):
        acc = None
        for k in range(0 if whole else 1, 2 * r + 3 - (0 if whole else 1)):
            part = a.narrow(dim, 2 * r + 2 - k, size) * t[k]
            acc = part if acc is None else acc.add_(part)
        return acc

    for a in range(2):
        for b in range(2):
            whole = bool(a or b)  # on the grid's whole points the window is one tap smaller each side
            rows = [conv(p, taps[4 * b + f], 1, w, whole) for f in range(4)]
            for k, (fx, fy) in enumerate(_NINE):
                out[k, a::2, b::2] = conv(rows[fx], taps[4 * a + fy], 0, h, whole)
    return out


def _third_order(d):
    fx, fy, fxx, fxy, fyy, fxxy, fxyy, fxxx, fyyy = d
    tx = fx * (2 * fxx * fxx + 2 * fxy * fxy) + fy * (2 * fxx * fxy + 2 * fyy * fxy) + 2 * fx * fy * fxxy \
        + fy * fy * fxyy + fx * fx * fxxx
    ty = fx * (2 * fxx * fxy + 2 * fyy * fxy) + fy * (2 * fyy * fyy + 2 * fxy * fxy) + 2 * fx * fy * fxyy \
        + fx * fx * fxxy + fy * fy * fyyy
    return tx, ty


def _sector(dx, dy):
    """Offsets (row, column) of the axis and the diagonal neighbour ahead, and the slope between them."""
    xmaj = dx.abs() >= dy.abs()
    sx, sy = torch.where(dx >= 0, 1, -1), torch.where(dy >= 0, 1, -1)
    zero = torch.zeros_like(sx)
    axis = (torch.where(xmaj, zero, sy), torch.where(xmaj, sx, zero))
    slope = torch.where(xmaj, dy.abs() / dx.abs(), dx.abs() / dy.abs())
    return axis, (sy, sx), slope


def _fit(f, ap, dp, am, dm, slope):
    """(is a maximum, s*, peak) of the parabola through the interpolated neighbours."""
    fp, fm = ap * (1 - slope) + dp * slope, am * (1 - slope) + dm * slope
    s = torch.sqrt(1 + slope * slope)
    A, B = (fm + fp - 2 * f) / (2 * s * s), (fp - fm) / (2 * s)
    at = -B / (2 * A)
    top = ((f > fm) & (f >= fp)) | ((f >= fm) & (f > fp))
    return top & (at.abs() <= math.sqrt(2.0)), at, A * at * at + B * at + f, A


def _keys(s):
    x = s.abs()
    near = (1.5 * x - 2.5) * x * x + 1
    far = ((-0.5 * x + 2.5) * x - 4) * x + 2
    return torch.where(x <= 1, near, torch.where(x < 2, far, torch.zeros_like(x)))


def _bicubic(plane, x, y):
    """Cubic convolution (a = -1/2) of a plane at (x, y), coordinates clamped to it."""
    h, w = plane.shape
    x0, y0 = x.floor(), y.floor()
    out = torch.zeros_like(x)
    for p in range(4):
        ii = (y0.long() - 1 + p).clamp(0, h - 1)
        for q in range(4):
            jj = (x0.long() - 1 + q).clamp(0, w - 1)
            out += plane[ii, jj] * _keys(x - x0 + 1 - q) * _keys(y - y0 + 1 - p)
    return out


#: How far (in gradient magnitude) two sides of a decision have to be apart for
#: 32-bit derivatives of pixels up to 255 to decide it the same way.
CLEAR = 5e-6


def _detect64(img, case):
    """(edgels, 2x-grid index, whether every decision is a clear one) of one image."""
    r = math.ceil(4 * case["sigma"])
    mode = case.get("mode", "grid")
    h, w = img.shape
    d = _dense9(img.double(), _taps64(torch.tensor(case["sigma"], dtype=torch.float64, device=DEV), r), r)
    M = torch.sqrt(d[0] ** 2 + d[1] ** 2)
    ok = (M > case.get("threshold", 2.0)) & ~((d[0].abs() < 1e-5) & (d[1].abs() < 1e-5))
    inner = torch.zeros_like(ok)
    inner[10:2 * h - 10, 10:2 * w - 10] = True
    i, j = torch.nonzero(ok & inner, as_tuple=True)
    at = [x[i, j] for x in d]
    m = M[i, j]
    dx, dy = _third_order(at) if mode == "normal" else (at[0], at[1])
    length = torch.sqrt(dx * dx + dy * dy)
    (ar, ac), (dr, dc), slope = _sector(dx, dy)
    near = [M[i + ar, j + ac], M[i + dr, j + dc], M[i - ar, j - ac], M[i - dr, j - dc]]
    keep, s, peak, _ = _fit(m, *near, slope)
    keep &= length > 0
    fp, fm = near[0] * (1 - slope) + near[1] * slope, near[2] * (1 - slope) + near[3] * slope
    clear = ((m - fp).abs() > CLEAR) | (fm - m > CLEAR)
    clear &= ((m - fm).abs() > CLEAR) | (fp - m > CLEAR)
    clear &= ((s.abs() - math.sqrt(2.0)).abs() * (2 * m - fp - fm).abs() > CLEAR) | ~((m > fp) & (m > fm))
    clear = bool(clear.all()) and not bool(((M - case.get("threshold", 2.0)).abs() < CLEAR).any())
    i, j, s, peak = i[keep], j[keep], s[keep], peak[keep]
    nx, ny = (dx / length)[keep], (dy / length)[keep]
    px, py = j + s * nx, i + s * ny
    tx, ty = _third_order([_bicubic(x, px, py) for x in d] if mode == "qad" else [x[keep] for x in at])
    edgels = torch.stack([(px - 1) / 2, (py - 1) / 2, torch.atan2(tx, -ty), peak.abs()], 1)
    return edgels, i * 2 * w + j, clear


def _derivs64(pad, r, i, j, taps, pairs):
    """Derivatives of an image at 2x-grid points, differentiable in the image and the taps."""
    n = 2 * r + 3
    a, b = i % 2, j % 2
    k = torch.arange(n, device=DEV)
    win = pad[(i // 2 + 2 * r + 2)[:, None, None] - k[None, :, None],
              (j // 2 + 2 * r + 2)[:, None, None] - k[None, None, :]]
    ends = ((k == 0) | (k == n - 1))[None, :] & ((a == 0) & (b == 0))[:, None]
    X = [torch.where(ends, 0.0, torch.where(b[:, None] == 1, taps[4 + f], taps[f])) for f in range(4)]
    Y = [torch.where(ends, 0.0, torch.where(a[:, None] == 1, taps[4 + f], taps[f])) for f in range(4)]
    return [torch.einsum("npq,nq,np->n", win, X[fx], Y[fy]) for fx, fy in pairs]


def _edgels64(img, sigma, index, r):
    """The edgels at given grid points, differentiable in img and sigma (the
    points and their sectors held fixed)."""
    h, w = img.shape
    i, j = index // (2 * w), index % (2 * w)
    taps = _taps64(sigma, r)
    pad = torch.nn.functional.pad(img, (r + 1,) * 4)
    d = _derivs64(pad, r, i, j, taps, _NINE)
    fx, fy = d[0], d[1]
    (ar, ac), (dr, dc), slope = _sector(fx, fy)
    m = torch.sqrt(fx * fx + fy * fy)
    near = []
    for r_, c_ in ((ar, ac), (dr, dc), (-ar, -ac), (-dr, -dc)):
        gx, gy = _derivs64(pad, r, i + r_, j + c_, taps, _NINE[:2])
        near.append(torch.sqrt(gx * gx + gy * gy))
    _, s, peak, _ = _fit(m, near[0], near[1], near[2], near[3], slope)
    tx, ty = _third_order(d)
    return torch.stack([(j + s * fx / m - 1) / 2, (i + s * fy / m - 1) / 2, torch.atan2(tx, -ty), peak.abs()], 1)


def _exact_gradients(case, seed):
    r = math.ceil(4 * case["sigma"])
    train = case["kind"] == "train"
    sigma = torch.tensor(case["sigma"], dtype=torch.float64, device=DEV, requires_grad=True)
    grads, gs, loss = [], 0.0, torch.zeros((), dtype=torch.float64, device=DEV)
    for img in _images(case, seed, disc=True):
        _, idx, _ = _detect64(img, case)
        x = img.double().requires_grad_(True)
        gi = torch.zeros_like(x)
        for part in idx.split(20000):  # the windows of 20,000 edgels at a time
            e = _edgels64(x, sigma, part, r)
            part_loss = _train_loss(e, *img.shape) if train else (e * _edgel_grads(part, e.detach())).sum()
            a, b = torch.autograd.grad(part_loss, [x, sigma])
            gi += a
            gs = gs + b
            loss += part_loss.detach()
        grads.append(gi)
    if not train:
        return {"grad_images": grads, "grad_sigma": gs}
    return {"loss": loss, "counts": None, "grad_images": torch.stack(grads), "grad_sigma": gs}


def _resize(E, n):
    """Corner-aligned bilinear resize to the grid 2^n times as fine."""
    h, w = E.shape
    H, W = (h - 1) * 2 ** n + 1, (w - 1) * 2 ** n + 1

    def line(size, fine):
        x = torch.arange(fine, dtype=torch.float64, device=DEV) * (size - 1) / (fine - 1)
        a = x.floor().long()
        return a, (a + 1).clamp(max=size - 1), x - a

    y0, y1, fy = line(h, H)
    x0, x1, fx = line(w, W)
    fy = fy[:, None]
    top, bottom = ((1 - fx) * E[y][:, x0] + fx * E[y][:, x1] for y in (y0, y1))
    return (1 - fy) * top + fy * bottom


def _hessian_angle(E):
    """Orientation estimate: triangle smoothing (radius 4, mirrored borders), second differences."""
    def smooth(a, dim):
        n = a.shape[dim]
        at = torch.arange(-4, n + 4, device=DEV)
        at = torch.where(at < 0, -at - 1, at)
        at = torch.where(at >= n, 2 * n - at - 1, at)
        a = a.index_select(dim, at)
        return sum(a.narrow(dim, 4 + k, n) * ((5 - abs(k)) / 25.0) for k in range(-4, 5))

    sm = smooth(smooth(E, 1), 0)
    oy, ox = torch.gradient(sm)
    oxx = torch.gradient(ox, dim=1)[0]
    oyy, oxy = torch.gradient(oy)
    return torch.remainder(torch.atan(oyy * -torch.sign(oxy) / (oxx + 1e-5)), math.pi)


def _correct64(E0, theta, case):
    """The corrected edgels and dense maps of one edge map."""
    n, sigma = case["interp_n"], case["sigma"]
    h0, w0 = E0.shape
    scale = 2 ** n
    E = _resize(E0, n) if n else E0
    h, w = E.shape
    th = _hessian_angle(E) if theta is None else torch.remainder(_resize(theta, n) if n else theta, math.pi)
    dx, dy = torch.cos(th), torch.sin(th)
    edge = 3 * scale
    ok = torch.zeros((h, w), dtype=torch.bool, device=DEV)
    ok[edge + 1:h - edge - 2, edge + 1:w - edge - 2] = True
    i, j = torch.nonzero(ok & (E > case["thresh"]), as_tuple=True)
    gx, gy, f = dx[i, j], dy[i, j], E[i, j]
    (ar, ac), (dr, dc), slope = _sector(gx, gy)
    keep, s, peak, A = _fit(f, E[i + ar, j + ac], E[i + dr, j + dc], E[i - ar, j - ac], E[i - dr, j - dc], slope)
    keep &= A.abs() >= 1e-16
    i, j, s, peak, gx, gy = (v[keep] for v in (i, j, s, peak, gx, gy))
    x, y = j + s * gx, i + s * gy
    # the circular separable convolutions
    r = math.ceil(4 * sigma)
    k = torch.arange(-r, r + 1, dtype=torch.float64, device=DEV)
    e = torch.exp(-k * k / (2 * sigma * sigma)) / math.sqrt(2 * math.pi)
    g = [e / sigma, -k * e / sigma ** 3, (k * k - sigma * sigma) * e / sigma ** 5]

    def conv(a, t, dim):
        return sum(torch.roll(a, q, dim) * t[q + r] for q in range(-r, r + 1))

    def at(a):
        return _bicubic(a, x, y)

    hx, hy = E * dx, E * dy
    eg, ed, edd = (conv(E, t, 1) for t in g)
    px, py = at(conv(ed, g[0], 0)), at(conv(eg, g[1], 0))
    pxx, pxy, pyy = at(conv(edd, g[0], 0)), at(conv(ed, g[1], 0)), at(conv(eg, g[2], 0))
    hxx, hyy, hxy = (at(conv(conv(a, g[p], 1), g[q], 0)) for a, p, q in ((hx, 1, 0), (hy, 0, 1), (hy, 1, 0)))
    vx, vy = at(hx), at(hy)
    fx, fy = px * hxx + pxx * vx + py * hxy + pxy * vy, px * hxy + pxy * vx + py * hyy + pyy * vy
    flat = torch.sqrt(fx * fx + fy * fy) < 1e-12
    angle = torch.where(flat, torch.atan2(gx, -gy), torch.atan2(fx, -fy))
    x, y = x / scale, y / scale
    if case["radius"] > 0 and len(x) >= 2:  # an edgel needs another within the radius
        reach = math.ceil(case["radius"] * scale + 3)
        who = torch.full((h + 2 * reach, w + 2 * reach), -1, dtype=torch.long, device=DEV)
        me = torch.arange(len(x), device=DEV)
        who[i + reach, j + reach] = me
        found = torch.zeros(len(x), dtype=torch.bool, device=DEV)
        for a in range(2 * reach + 1):
            for b in range(2 * reach + 1):
                o = who[i + a, j + b]
                hit = (x - x[o]) ** 2 + (y - y[o]) ** 2 <= case["radius"] ** 2
                found |= hit & (o >= 0) & (o != me)
        x, y, angle, peak = x[found], y[found], angle[found], peak[found]
    edgels = torch.stack([x, y, angle, peak.abs()], 1)

    def away(v, size):  # round half away from zero, into the map
        return torch.floor(v + 0.5).clamp(0, size - 1).long()

    spot = away(y, h0) * w0 + away(x, w0)
    last = torch.full((h0 * w0,), -1, dtype=torch.long, device=DEV)
    last.scatter_reduce_(0, spot, torch.arange(len(x), device=DEV), "amax")  # later edgels win
    some = last >= 0
    dense = [torch.where(some, edgels[:, c][last.clamp(min=0)], 0.0).reshape(h0, w0) if len(x)
             else torch.zeros((h0, w0), dtype=torch.float64, device=DEV) for c in (3, 2)]
    return edgels, dense


def _in_buffer(edgels, rows):
    """A list at the head of a buffer of zeros."""
    return torch.cat([edgels, torch.zeros((rows - len(edgels), 4), dtype=torch.float64, device=DEV)])


def exact(case, seed):
    """run's outputs in 64 bits.  A list has them only where every decision of
    its image is a clear one: decided the other way, one edgel more or less
    moves all later ones to another place.  Of the millions of decisions of a
    stream's, a graph's or a host batch's images some never are."""
    if case["kind"] in ("train", "adjoint"):
        return _exact_gradients(case, seed)
    if case["kind"] == "maps":
        maps, thetas = _ridge_maps(case, seed)
        res = [_correct64(E.double(), None if thetas is None else thetas[k].double(), case) for k, E in enumerate(maps)]
        return {"edgels": None, "counts": None, "TO_E": [d[0] for _, d in res], "TO_O": [d[1] for _, d in res]}
    if case["how"] != "call":
        return None
    lists = []
    for im in _images(case, seed):
        edgels, _, clear = _detect64(im, case)
        lists.append(_in_buffer(edgels, _capacity(*im.shape)) if clear else None)
    return {"edgels": lists, "index": None, "counts": None} if any(v is not None for v in lists) else None
