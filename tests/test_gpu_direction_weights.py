"""A pixel's estimated direction, which weights the correction of the edgels
around it, does not depend on whether the pixel itself lies above the
threshold: the edgels that two thresholds have in common are the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [1.0, 2.0])
@pytest.mark.parametrize("shape", [(224, 224), (131, 190)])
def test_directions_do_not_depend_on_the_threshold(detector, toed, shape, sigma):
    rng = np.random.default_rng(11)
    E = np.clip(0.05 + 0.5 * rng.random(shape), 0, 1).astype(np.float32)  # above 0.02 everywhere, above 0.4 in every tile
    lists = []
    for thresh in (0.4, 0.02):
        r = detector.subpix_to_correct_batch([torch.as_tensor(E).cuda()], thresh=thresh, sigma=sigma, nbr_radius=0.0,
                                             out_dtype=toed.TOED_F64)[0]
        lists.append({tuple(e[[0, 1]]): tuple(e[[2, 3]]) for e in r["edgels"].cpu().numpy()})
    few, many = lists
    assert len(few) > 300 and len(many) > 1.2 * len(few)
    assert all(many.get(at) == few[at] for at in few)
