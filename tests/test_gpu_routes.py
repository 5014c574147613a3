"""Both sides of each dispatch rule give the same results: the TO correction's
orientation estimate in integers and in double-floats, its dense maps, host
batches in one pipeline and in two, 8-bit rows from any alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _subpix(det, toed, E, thresh):
    return det.subpix_to_correct_batch([torch.as_tensor(E).cuda()], thresh=thresh, sigma=2.0, nbr_radius=2.0,
                                       out_dtype=toed.TOED_F64)[0]


@pytest.mark.parametrize("shape", [(33, 31), (97, 130), (64, 251)])
def test_orientation_in_integers_and_double_floats(detector, synth, toed, shape):
    """The integers serve tiles whose largest value is at most 256 times the
    threshold: with thresh 1e-3 a map of ridges near 1 takes the double-floats.
    Each edgel found above 0.1 is found there too (more neighbours isolate
    fewer); both estimates hold 2^-41, positions and angles FP32 offsets."""
    E = synth.ridge_map(*shape, seed=61, n_curves=5).astype(np.float32)
    a = _subpix(detector, toed, E, 0.1)["edgels"].cpu().numpy()
    b = _subpix(detector, toed, E, 1e-3)["edgels"].cpu().numpy()
    assert len(a) > 20
    from scipy.spatial import cKDTree
    d, j = cKDTree(b[:, :2]).query(a[:, :2])
    assert d.max() <= 1e-5
    turn = np.abs(np.angle(np.exp(1j * (a[:, 2] - b[j, 2]))))
    assert turn.max() <= 1e-5 and np.abs(a[:, 3] - b[j, 3]).max() <= 1e-5


@pytest.mark.parametrize("shape", [(64, 251), (97, 130), (64, 96)])
def test_dense_maps_hold_the_list(detector, synth, toed, shape):
    """Each pixel holds the last edgel of the list that rounds to it."""
    E = synth.ridge_map(*shape, seed=63, n_curves=6).astype(np.float32)
    r = _subpix(detector, toed, E, 0.1)
    want = np.zeros((2, *shape))
    edgels = r["edgels"].cpu().numpy()
    assert len(edgels) > 20
    x = np.clip(np.floor(edgels[:, 0] + 0.5).astype(int), 0, shape[1] - 1)
    y = np.clip(np.floor(edgels[:, 1] + 0.5).astype(int), 0, shape[0] - 1)
    for k in range(len(edgels)):
        want[:, y[k], x[k]] = edgels[k, 3], edgels[k, 2]
    np.testing.assert_array_equal(r["TO_E"].cpu().numpy(), want[0])
    np.testing.assert_array_equal(r["TO_O"].cpu().numpy(), want[1])
    f = detector.subpix_to_correct_batch([torch.as_tensor(E).cuda()], thresh=0.1, sigma=2.0, nbr_radius=2.0)[0]
    np.testing.assert_array_equal(f["TO_E"].cpu().numpy(), want[0].astype(np.float32))
    np.testing.assert_array_equal(f["TO_O"].cpu().numpy(), want[1].astype(np.float32))


@pytest.mark.parametrize("f64,index", [(False, True), (True, True), (True, False)])
def test_host_batch_in_two_pipelines(toed, synth, f64, index):
    """12.6 Mpixel: 45 % of the batch (over 4 Mi pixels) is left to a second launch."""
    det = toed.Detector(0)
    base = synth.shapes_image(1500, 1400, seed=64, dtype=np.float32).image
    host = [torch.as_tensor(np.roll(base, 37 * k, axis=1).copy()).pin_memory() for k in range(6)]
    dt = toed.TOED_F64 if f64 else toed.TOED_F32
    ref = det.detect_batch([im.cuda() for im in host], sigma=1.5, out_dtype=dt)
    outs = det.alloc_host_outputs([tuple(im.shape) for im in host], out_dtype=dt, index=index)
    prm = toed.make_params(1.5, 0, 2.0, 10, dt)
    for _ in range(2):
        det.detect_host(host, outs, prm)
        for r, o in zip(ref, outs):
            n = int(o["count"].item())
            assert n == r["count"] > 0
            assert torch.equal(o["edgels"][:n], r["edgels"].cpu())
            if index:
                assert torch.equal(o["index"][:n], r["index"].cpu())


@pytest.mark.parametrize("start", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", [(50, 61), (97, 150)])
def test_8bit_rows_from_any_alignment(toed, synth, shape, start):
    det = toed.Detector(0)
    H, W = shape
    im = torch.as_tensor(synth.shapes_image(H, W, seed=65, dtype=np.uint8).image).cuda()
    buf = torch.zeros((H, W + 7), dtype=torch.uint8, device="cuda")
    buf[:, start:start + W] = im
    a, b = det.detect_batch([im, buf[:, start:start + W]], sigma=1.5)
    assert a["count"] == b["count"] > 0 and torch.equal(a["edgels"], b["edgels"]) and torch.equal(a["index"], b["index"])


@pytest.mark.parametrize("side,interp_n", [(1024, 0), (512, 1)])
def test_segment_tiles_shared_out_or_whole(detector, synth, toed, side, interp_n):
    """A map's segment tiles (isolation; dense maps of a work grid) are shared out over CTAs alone, taken whole among ten maps (320 tiles)."""
    E = [torch.as_tensor(synth.ridge_map(side, side, seed=66 + k, n_curves=9).astype(np.float32)).cuda() for k in range(10)]
    together = detector.subpix_to_correct_batch(E, thresh=0.1, sigma=1.0, nbr_radius=2.0, interp_n=interp_n)
    for k in (0, 9):
        alone = detector.subpix_to_correct_batch([E[k]], thresh=0.1, sigma=1.0, nbr_radius=2.0, interp_n=interp_n)[0]
        assert alone["count"] == together[k]["count"] > 100
        for name in ("edgels", "TO_E", "TO_O"):
            assert torch.equal(alone[name], together[k][name])
