"""The staging area has room for every edgel of lists that fit, however the
warps' reservations fall: capacity equal to the count, few edgels a warp and
step, so that a warp drops the rest of its reservation block again and again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threshold", [2.5, 3.0])
def test_exact_capacity_loses_nothing(toed, threshold):
    gen = torch.Generator(device="cuda").manual_seed(5)
    im = (128 + 25 * torch.randn(8192, 8192, generator=gen, device="cuda")).contiguous()
    prm = toed.make_params(2.0, 0, threshold)

    def lists(capacity):
        det = toed.Detector(0)
        out = det.alloc_outputs([im.shape], capacity=capacity)[0]
        out["index"].fill_(-1)
        det.detect_into([im], [out], prm)
        n, flags = int(out["count"].item()), det.flags()
        det.close()
        return n, flags, out

    n, flags, roomy = lists(im.numel())
    assert flags == 0 and n > 2_000_000
    m, flags, exact = lists(n)
    assert flags == 0 and m == n
    assert torch.equal(exact["index"], roomy["index"][:n])
    assert torch.equal(exact["edgels"].view(torch.int32), roomy["edgels"][:n].view(torch.int32))
