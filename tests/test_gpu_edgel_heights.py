"""The edgel kernel's tiles are 24, 48, 96 or 192 rows high by the size of the
launch: images whose last rows fall around each of these edges give the same
lists bit for bit beside companions that call for each height."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HEIGHTS = [23, 24, 25, 47, 48, 49, 95, 96, 97, 191, 192, 193]
WIDTHS = [61, 40, 90, 31]


def _height(sizes):
    """The tile height for images of the sizes: eight tiles an SM, halved from 192 to 24 at least."""
    rows = sum((w + 29) // 30 * h for h, w in sizes)
    t, sms = 192, torch.cuda.get_device_properties(0).multi_processor_count
    while t > 24 and rows < t * 8 * sms:
        t //= 2
    return t


@pytest.mark.parametrize("mode", ["grid", "qad", "normal"])
@pytest.mark.parametrize("dtype", [np.float32, np.uint8])
def test_every_height_gives_the_same_lists(toed, mode, dtype):
    kw = {"grid": {}, "qad": {"orientation": toed.TOED_ORI_QAD}, "normal": {"nms_direction": toed.TOED_NMS_TO_NORMAL}}[mode]
    rng = np.random.default_rng(3)
    ims = []
    for k, h in enumerate(HEIGHTS):
        x = np.clip(rng.normal(128, 25, (h, WIDTHS[k % 4])), 0, 255)
        ims.append(torch.as_tensor((np.rint(x) if dtype == np.uint8 else x).astype(dtype)).cuda())
    sizes = [tuple(im.shape) for im in ims]
    det = toed.Detector(0)
    per_row = -(-8 * torch.cuda.get_device_properties(0).multi_processor_count // 137)  # of 137 strips, 8 tiles an SM
    base, seen = None, []
    for rows in (0, 52, 100, 196):
        more = [torch.zeros((rows * per_row, 4096), dtype=ims[0].dtype, device="cuda")] if rows else []  # no edgels
        seen.append(_height(sizes + [tuple(m.shape) for m in more]))
        res = det.detect_batch(more + ims, sigma=1.5, threshold=0.5, border=2, capacity=40000, **kw)[len(more):]
        lists = [(r["edgels"].view(torch.int32), r["index"]) for r in res]
        assert sum(len(i) for _, i in lists) > 3000
        base = base or lists
        for (e, i), (f, j), s in zip(base, lists, sizes):
            assert torch.equal(i, j) and torch.equal(e, f), (s, seen[-1])
    assert seen == [24, 48, 96, 192]
