"""Host batches: one detection launch for a batch of up to 64 page-locked
images, whatever its size (so the shape tuned for such a batch serves it);
every layout of outputs, images without edgels and a lost copy in large batches."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(synth, sizes):
    """Page-locked float32 images of the sizes, the fourth without edgels."""
    base = synth.shapes_image(1500, 1400, seed=64, dtype=np.float32).image
    out = []
    for k, (h, w) in enumerate(sizes):
        im = np.roll(np.tile(base, (2, 2)), 37 * k, axis=1)[:h, :w]
        out.append(torch.as_tensor(np.full((h, w), 90, np.float32) if k == 3 else np.ascontiguousarray(im)).pin_memory())
    return out


# 26.8 Mpixel, the larger part behind the first half; sizes uneven, one image empty
SIZES = [(1500, 1400), (900, 2100), (2011, 1301), (1400, 1500), (2048, 2048), (1203, 907), (2048, 2048), (1801, 2001), (640, 1111),
         (1500, 1400)]


@pytest.mark.parametrize("pin", [True, False])
@pytest.mark.parametrize("f64", [False, True])
def test_one_launch_for_a_large_batch(toed, synth, pin, f64):
    det = toed.Detector(0)
    host = _batch(synth, SIZES)
    dt = toed.TOED_F64 if f64 else toed.TOED_F32
    ref = det.detect_batch([im.cuda() for im in host], sigma=1.5, out_dtype=dt)
    outs = det.alloc_host_outputs(SIZES, capacity=400_000, out_dtype=dt, index=True, pin=pin)
    prm = toed.make_params(1.5, 0, 2.0, 10, dt)
    for _ in range(2):
        det.profile_begin()
        det.detect_host(host, outs, prm)
        assert det.profile_end()[1] == 1
        for k, (r, o) in enumerate(zip(ref, outs)):
            n = int(o["count"].item())
            assert n == r["count"] and (n == 0 if k == 3 else n > 1000)
            assert torch.equal(o["edgels"][:n], r["edgels"].cpu())
            assert torch.equal(o["index"][:n], r["index"].cpu())


def _child(body, **env):
    """Runs `body` in a process of its own (the library reads the injections' variables there)."""
    code = f"""
import os, sys, time
sys.path.insert(0, {os.path.dirname(os.path.abspath(__file__))!r})
from conftest import load_package
toed = load_package()
import torch
from test_gpu_host_launch import SIZES, _batch
import importlib
synth = importlib.import_module("toed_gb300.synth")
det = toed.Detector(0)
prm = toed.make_params(1.5)
host = _batch(synth, SIZES)
""" + body
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=dict(os.environ, **env))
    assert r.returncode == 0 and "OK" in r.stdout, r.stderr[-3000:]


def test_lost_copy_in_a_large_batch(toed):
    """Group 7's ready flag is withheld on the host: the call returns the
    time-out within its bound, the other images keep their edgels, and the next
    call succeeds."""
    _child("""
ref = [r["count"] for r in det.detect_batch([im.cuda() for im in host], sigma=1.5)]
outs = det.alloc_host_outputs(SIZES, capacity=400000)
os.environ["TOED_TEST_WITHHOLD_READY"] = "7"
os.environ["TOED_TEST_READY_SPINS"] = "20000"
t0 = time.time()
try:
    det.detect_host(host, outs, prm)
    raise SystemExit("no time-out")
except toed.ToedError as e:
    assert e.status == toed.TOED_ERR_TIMEOUT, e
assert time.time() - t0 < 5
got = [int(o["count"].item()) for o in outs]
assert got[:7] == ref[:7] and got[7] == 0, (got, ref)
del os.environ["TOED_TEST_WITHHOLD_READY"], os.environ["TOED_TEST_READY_SPINS"]
det.detect_host(host, outs, prm)
assert [int(o["count"].item()) for o in outs] == ref
print("OK")
""")


def test_one_group_asked_for_crosses_in_several(toed):
    """chunks = 1: more groups are used, so that detection starts before the
    last pixel is in -- seen by withholding the second group's flag."""
    _child("""
outs = det.alloc_host_outputs(SIZES, capacity=400000)
try:
    det.detect_host(host, outs, prm, chunks=1)
    raise SystemExit("one group")
except toed.ToedError as e:
    assert e.status == toed.TOED_ERR_TIMEOUT, e
print("OK")
""", TOED_TEST_WITHHOLD_READY="1", TOED_TEST_READY_SPINS="4096")


@pytest.mark.parametrize("chunks", [1, 5])
def test_no_device_memory_for_the_pixels(toed, chunks):
    """Page-locked images are read in place when device memory for them cannot
    be had: float32 and 8-bit, rows off 16-byte boundaries, lists as ever."""
    _child(f"""
wide = torch.zeros((1400, 1503), dtype=torch.float32).pin_memory()
wide[:, 1:1501] = host[1][:900].repeat(2, 1)[:1400, :1500]
ims = host + [wide[:, 1:1501], host[4].round().to(torch.uint8).pin_memory(), host[5].round().to(torch.uint8).pin_memory()]
ref = det.detect_batch([im.contiguous().cuda() for im in ims], sigma=1.5)
ref = [(r["count"], r["edgels"].cpu(), r["index"].cpu()) for r in ref]
outs = det.alloc_host_outputs([tuple(im.shape) for im in ims], capacity=400000, index=True)
for k in range(2):
    det.detect_host(ims, outs, prm, chunks={chunks})
    for (n, e, i), o in zip(ref, outs):
        assert int(o["count"].item()) == n and torch.equal(o["edgels"][:n], e) and torch.equal(o["index"][:n], i)
det.close()
torch.cuda.empty_cache()
# a fresh context, a threshold that nothing reaches: no staging for the 107 MB of pixels is held
det = toed.Detector(0)
outs = det.alloc_host_outputs([tuple(im.shape) for im in ims], capacity=2000)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
det.detect_host(ims, outs, toed.make_params(1.5, threshold=1e6), chunks={chunks})
held = free - torch.cuda.mem_get_info()[0]
assert held < 60e6, held
print("OK")
""", TOED_TEST_NO_STAGING="1")
