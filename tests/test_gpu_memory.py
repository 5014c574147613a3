"""A context holds the memory that its calls use and no more: detection its
staging records, segments and scan words, the TO correction its records, indices
and per-pixel planes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _held(call):
    """Device memory that `call` takes outside torch's allocator."""
    torch.cuda.synchronize()
    free, own = torch.cuda.mem_get_info()[0], torch.cuda.memory_reserved()
    call()
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0] - (torch.cuda.memory_reserved() - own)


def _detection(det, toed, rows):
    im = torch.zeros((512, 512), device="cuda")
    outs = det.alloc_outputs([im.shape], capacity=rows)
    return lambda: det.detect_into([im], outs, toed.make_params(1.5))


def _correction(det, side, **kw):
    E = torch.zeros((side, side), device="cuda")
    E[side // 2] = 0.5
    return lambda: det.subpix_to_correct_batch([E], thresh=0.1, **kw)


def test_detection(toed):
    _detection(toed.Detector(0), toed, 1000)()  # the kernels' code is loaded
    rows = 16_000_000
    det = toed.Detector(0)
    # 32 bytes a record, 64/57 of the capacity; a block of 64 records a warp of the chip
    assert _held(_detection(det, toed, rows)) <= 32 * rows * 64 // 57 + 40 * MB
    det.close()
    det = toed.Detector(0)
    assert _held(lambda: det.reserve(1 << 20, rows, 1)) <= 32 * rows * 64 // 57 + 48 * MB


@pytest.mark.parametrize("interp_n", [0, 1])
def test_correction(toed, interp_n):
    _correction(toed.Detector(0), 64, interp_n=interp_n)()
    side = 4096 >> interp_n
    px = ((side - 1 << interp_n) + 1) ** 2
    # a record of 32 bytes, an index and a flag for each pixel of the capacity;
    # a direction (8) and an id (4) a pixel; on a work grid its map (8) and winners (4)
    per_px = 32 + 4 + 1 + 8 + 4 + (12 if interp_n else 0)
    assert _held(_correction(toed.Detector(0), side, interp_n=interp_n)) <= per_px * px + 24 * MB


def test_noalloc_scratch_is_what_its_comment_says(toed):
    """The array holds 32 bytes an edgel and 12 a segment: 12 MB."""
    import os
    import re
    src = open(os.path.join(os.path.dirname(toed.__file__), "csrc", "toed_noalloc.cu")).read()
    assert not re.search(r"kOff(Idx|Tiles|Base)", src) and "about 12 MB" in src
