"""The adjoint's window evaluation at the sizes where it can go wrong: each
staging route (aligned groups of float pixels, 8-bit pixels), windows inside
and across the image's border, images smaller than a window, rows that start
anywhere in a group of four, both parities in one round, chunks of several
images.  Against the FP64 frozen-selection restatement differentiated by torch
autograd; the cotangents are those of the clear edges (strength above 10),
whose peak fit magnifies the FP32 sums' 1e-6 by at most about a hundred."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 1e-4


@pytest.mark.parametrize("radius,shape,start,dtype", [
    (1, (33, 41), 0, "f32"),
    (2, (40, 35), 1, "f32"),
    (3, (64, 61), 3, "f32"),
    (5, (47, 90), 2, "f32"),
    (8, (19, 23), 1, "f32"),   # smaller than the window
    (8, (97, 130), 3, "f32"),
    (8, (97, 130), 1, "u8"),
    (9, (70, 66), 2, "f32"),
    (12, (25, 27), 0, "f32"),
    (12, (75, 64), 1, "u8"),
])
def test_adjoint_windows(toed, synth, radius, shape, start, dtype):
    from oracle import frozen
    det = toed.Detector(0)
    H, W = shape
    sigma = max(0.7, radius / 4)
    views = []
    for k in range(2):  # one buffer's columns start .. start + W: rows begin anywhere in a group
        im = synth.shapes_image(H, W, seed=8200 + k, dtype=np.float32, ellipses_only=True, n_shapes=3,
                                radius_range=(5, 20), scale_to_base=False).image
        im = np.clip(im + np.random.default_rng(8300 + k).normal(0.0, 2.0, im.shape), 0, 255)
        buf = torch.zeros((H, W + 5), dtype=torch.uint8 if dtype == "u8" else torch.float32, device="cuda")
        buf[:, start:start + W] = torch.as_tensor(np.rint(im) if dtype == "u8" else im).to(buf.dtype).cuda()
        views.append(buf[:, start:start + W])
    res = det.detect_batch(views, sigma=sigma, radius=radius, border=4)
    assert sum(r["index"].numel() for r in res) > 20
    g_out = [torch.stack([torch.cos(0.37 * r["index"].double() + k) for k in range(4)], 1).float()
             * (r["edgels"][:, 3:] > 10) for r in res]
    grads, gs = det.backward_batch(views, [r["index"] for r in res], g_out, sigma=sigma, radius=radius)

    s64 = torch.tensor(sigma, dtype=torch.float64, requires_grad=True)
    x64 = [v.double().cpu().requires_grad_(True) for v in views]
    loss = sum((frozen.edgel_outputs(x, s64, r["index"].cpu(), radius) * g.double().cpu()).sum()
               for x, r, g in zip(x64, res, g_out))
    ref = torch.autograd.grad(loss, x64 + [s64])
    got = torch.cat([g.double().cpu().flatten() for g in grads])
    want = torch.cat([g.flatten() for g in ref[:-1]])
    assert float((got - want).norm()) <= REL * float(want.norm())
    # dL/dsigma: a sum of terms of the order of one, one an edgel, that may cancel
    used = sum(int((g.abs().sum(1) > 0).sum()) for g in g_out)
    assert abs(float(gs) - float(ref[-1])) <= REL * (abs(float(ref[-1])) + used)
