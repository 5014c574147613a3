"""The edgel kernel's tiles: heights from 12 to 192 rows by the size of the
launch, pixels staged by TMA or by loads, more edgels than a chunk holds,
strip and tile remainders -- every cut of the work gives the same list bit for
bit, and the list is the oracle's."""
import numpy as np
import pytest
import torch

from conftest import compare_edgels

pytestmark = pytest.mark.gpu

# rows around a tile's edges (12 .. 192), columns around a strip's (30)
SIZES = [(1, 40), (11, 29), (12, 30), (13, 31), (25, 61), (191, 90), (192, 91), (193, 97), (385, 64)]


def _detect(det, images, sigma, thr, **kw):
    res = det.detect_batch(images, sigma=sigma, threshold=thr, **kw)
    return [(r["edgels"].clone(), r["index"].clone()) for r in res]


def _noise(h, w, seed, dtype):
    rng = np.random.default_rng(seed)
    img = np.clip(rng.normal(128, 25, (h, w)), 0, 255)
    return torch.as_tensor(img.astype(dtype) if dtype == np.float32 else np.rint(img).astype(np.uint8)).cuda()


@pytest.mark.parametrize("mode", ["grid", "qad", "normal"])
@pytest.mark.parametrize("sigma,dtype", [(1.0, np.float32), (2.0, np.uint8)])
def test_every_cut_gives_the_same_list(detector, toed, mode, sigma, dtype):
    kw = {"grid": {}, "qad": {"orientation": toed.TOED_ORI_QAD}, "normal": {"nms_direction": toed.TOED_NMS_TO_NORMAL}}[mode]
    det = toed.Detector(0)
    imgs = [_noise(h, w, 7 * h + w, dtype) for h, w in SIZES]
    alone = [_detect(det, [x], sigma, 0.5, **kw)[0] for x in imgs]  # the smallest tiles
    # a batch long enough for the tallest tiles (the big image holds no edgels)
    big = torch.zeros((2000, 4096), dtype=imgs[0].dtype, device="cuda")
    tall = _detect(det, [big] + imgs, sigma, 0.5, capacity=200 * 100 * 4, **kw)[1:]
    # rows that start off 16-byte boundaries: loads instead of TMA
    shifted = []
    for x in imgs:
        buf = torch.zeros((x.shape[0], x.shape[1] + 3), dtype=x.dtype, device="cuda")
        buf[:, 1:1 + x.shape[1]] = x
        shifted.append(buf[:, 1:1 + x.shape[1]])
    loads = _detect(det, shifted, sigma, 0.5, **kw)
    assert sum(len(i) for _, i in alone) > 5000
    for k, (e, i) in enumerate(alone):
        for other in (tall, loads):
            assert torch.equal(i, other[k][1]), (SIZES[k], len(i), len(other[k][1]))
            assert torch.equal(e.view(torch.int32), other[k][0].view(torch.int32)), SIZES[k]


@pytest.mark.parametrize("orientation", ["grid", "qad"])
def test_dense_tiles_vs_oracle(detector, oracle, toed, orientation):
    """More edgels in a tile than a chunk holds (pure noise, a low threshold)."""
    img = _noise(900, 1300, 5, np.float32)
    kw = {"orientation": toed.TOED_ORI_QAD} if orientation == "qad" else {}
    (e, i), = _detect(toed.Detector(0), [img], 1.0, 1.0, **kw)
    ref = oracle.detect(img.double().cpu().numpy(), 1.0, threshold=1.0, orientation=orientation)
    m = compare_edgels(ref["edges"], ref["index"], e.double().cpu().numpy(), i.cpu().numpy())
    assert m["n_common"] > 100000 and m["agreement"] >= 0.999, m
    assert m["pos_p99"] <= 1e-3 and m["ori_p99"] <= 1e-4, m
