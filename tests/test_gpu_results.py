"""Each image's results are its own: no storage, and no autograd version
counter, is shared with another image's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _own(tensors, rows):
    """Every tensor's storage belongs to it alone and holds at most `rows` of it."""
    assert len({t.untyped_storage().data_ptr() for t in tensors}) == len(tensors)
    for t, r in zip(tensors, rows):
        assert t.untyped_storage().nbytes() <= r * t.element_size() * t[0].numel()
        assert not t._is_view() or t._base is None or t._base.untyped_storage().nbytes() == t.untyped_storage().nbytes()


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("n", [1, 3])
def test_detect_batch(toed, synth, n, f64):
    sizes = [(97, 150), (211, 160), (130, 97)][:n]
    ims = [torch.as_tensor(synth.shapes_image(h, w, seed=40 + k, dtype=np.float32).image).cuda() for k, (h, w) in enumerate(sizes)]
    res = toed.Detector(0).detect_batch(ims, sigma=1.5, out_dtype=toed.TOED_F64 if f64 else toed.TOED_F32)
    assert all(r["count"] > 20 for r in res)
    _own([r["edgels"] for r in res] + [r["index"] for r in res], [4 * h * w for h, w in sizes] * 2)
    if n > 1:  # an edit of one list in place leaves the others as autograd saved them
        x = torch.ones(4, device="cuda", requires_grad=True)
        loss = (x * res[0]["edgels"].to(x.dtype)).sum()
        res[1]["edgels"].zero_()
        loss.backward()


def test_subpix_maps(detector, synth):
    E = [torch.as_tensor(synth.ridge_map(90 + 31 * k, 140, seed=66 + k, n_curves=4).astype(np.float32)).cuda() for k in range(3)]
    res = detector.subpix_to_correct_batch(E, thresh=0.1)
    assert all(r["count"] > 20 for r in res)
    _own([r["edgels"] for r in res], [e.numel() for e in E])
    _own([r[k] for r in res for k in ("TO_E", "TO_O")], [e.shape[0] for e in E for _ in range(2)])


def test_bad_images_are_refused(detector):
    for bad in (torch.zeros(5, device="cuda"), torch.zeros((4, 4), dtype=torch.float64, device="cuda"), torch.zeros((4, 4)),
                torch.zeros((8, 8), device="cuda").t()[:, ::2]):
        with pytest.raises(ValueError):
            detector.detect_batch([bad])
