"""The adjoint on images packed one behind the other with nothing between them,
starting anywhere in a group of four pixels: the windows at a storage's first
and last pixels, whose group of four is shared with the neighbour, come from
single pixels.  Against the FP64 frozen-selection restatement differentiated by
torch autograd, cotangents of the clear edges, as for the other windows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 1e-4


def _corners(h, w, radius, seed):
    """A disc around each corner, where the first and last windows lie, and one in the middle."""
    y, x = np.mgrid[0:h, 0:w]
    im = np.full((h, w), 90.0)
    rad = 1.2 * radius + 2  # its nearest edgels' windows reach the corner
    for cy, cx in ((0, 0), (h, w), (0, w), (h, 0), (h / 2, w / 2)):
        im += 110 / (1 + np.exp(2 * (np.hypot(y + 0.5 - cy, x + 0.5 - cx) - rad)))
    return np.clip(im + np.random.default_rng(seed).normal(0, 1.0, im.shape), 0, 255)


@pytest.mark.parametrize("radius,start,dtype", [(2, 1, "f32"), (4, 2, "f32"), (6, 3, "f32"), (6, 1, "u8"), (8, 3, "u8"), (12, 1, "f32")])
def test_packed_images(toed, radius, start, dtype):
    from oracle import frozen
    sigma = max(0.7, radius / 4)
    sizes = [(57, 63), (48, 51), (71, 45)]
    ims = [_corners(h, w, radius, 70 + k) for k, (h, w) in enumerate(sizes)]
    if dtype == "u8":
        ims = [np.rint(im) for im in ims]
    flat = torch.zeros(start + sum(h * w for h, w in sizes), dtype=torch.uint8 if dtype == "u8" else torch.float32, device="cuda")
    views, at = [], start
    for im, (h, w) in zip(ims, sizes):
        views.append(flat[at:at + h * w].view(h, w))
        views[-1].copy_(torch.as_tensor(im))
        at += h * w
    det = toed.Detector(0)
    res = det.detect_batch(views, sigma=sigma, radius=radius, border=2)
    g_out = [torch.stack([torch.cos(0.37 * r["index"].double() + k) for k in range(4)], 1).float()
             * (r["edgels"][:, 3:] > 10) for r in res]
    first = last = 0  # used edgels whose window holds the storage's first, or last, pixel, in a shared group
    pos = start
    for r, g, (h, w) in zip(res, g_out, sizes):
        i, j = r["index"] // (2 * w) // 2, r["index"] % (2 * w) // 2
        used = g.abs().sum(1) > 0
        assert int(used.sum()) > 40
        first += int((used & (i <= radius + 2) & (j <= radius + 2)).sum()) if pos % 4 else 0
        pos += h * w
        last += int((used & (i >= h - radius - 3) & (j >= w - radius - 3)).sum()) if pos % 4 else 0
    assert first > 0 and last > 0
    grads, gs = det.backward_batch(views, [r["index"] for r in res], g_out, sigma=sigma, radius=radius)
    s64 = torch.tensor(sigma, dtype=torch.float64, requires_grad=True)
    x64 = [v.double().cpu().requires_grad_(True) for v in views]
    loss = sum((frozen.edgel_outputs(x, s64, r["index"].cpu(), radius) * g.double().cpu()).sum()
               for x, r, g in zip(x64, res, g_out))
    ref = torch.autograd.grad(loss, x64 + [s64])
    for got, want in zip(grads, ref):
        assert float((got.double().cpu() - want).norm()) <= REL * float(want.norm())
    used = sum(int((g.abs().sum(1) > 0).sum()) for g in g_out)
    assert abs(float(gs) - float(ref[-1])) <= REL * (abs(float(ref[-1])) + used)
