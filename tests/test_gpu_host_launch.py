"""Host batches of page-locked images: one detection launch, or two where the
rule says so; every layout of outputs, images without edgels and lost copies in
large batches; one group asked for; no device memory for the pixels."""
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


# 57.6 Mpixel in 35 images, uneven, one of the first and one of the second part empty (see MANY_EMPTY)
MANY = [(1100 + 37 * (k % 7), 1300 + 29 * (k % 5)) for k in range(35)]
MANY_EMPTY = (3, 30)


def _many(synth):
    out = _batch(synth, MANY)
    out[30] = torch.full(MANY[30], 55.0).pin_memory()
    return out


@pytest.mark.parametrize("pin", [True, False])
@pytest.mark.parametrize("f64", [False, True])
def test_two_launches_for_many_images(toed, synth, pin, f64):
    """At the rule's lines: 35 float32 images of 57.6 Mpixel take two launches,
    31 of them, a wider filter or less than 56 Mpixel one; the lists are the
    device batch's, also at a shape tuned for the whole batch."""
    det = toed.Detector(0)
    host = _many(synth)
    assert sum(im.numel() for im in host) > 56e6
    dt = toed.TOED_F64 if f64 else toed.TOED_F32
    outs = det.alloc_host_outputs(MANY, capacity=200_000, out_dtype=dt, index=True, pin=pin)

    def launches(n, sigma, images=None):
        images = images or host[:n]
        det.profile_begin()
        det.detect_host(images, outs[:n], toed.make_params(sigma, 0, 2.0, 10, dt))
        return det.profile_end()[1]

    def same(n, sigma):
        ref = det.detect_batch([im.cuda() for im in host[:n]], sigma=sigma, out_dtype=dt)
        for k, (r, o) in enumerate(zip(ref, outs)):
            m = int(o["count"].item())
            assert m == r["count"] and (m == 0 if k in MANY_EMPTY else m > 1000)
            assert torch.equal(o["edgels"][:m], r["edgels"].cpu())
            assert torch.equal(o["index"][:m], r["index"].cpu())

    assert launches(35, 1.5) == 2
    same(35, 1.5)
    assert launches(35, 1.0) == 2
    same(35, 1.0)
    assert launches(31, 1.5) == 1 and launches(33, 1.5) == 1 and launches(35, 1.6) == 1
    same(35, 1.6)
    small = [im[:, 200:].contiguous().pin_memory() for im in host]
    assert launches(35, 1.5, [im.round().to(torch.uint8).pin_memory() for im in host]) == 1
    assert sum(im.numel() for im in small) < 56e6 and launches(35, 1.5, small) == 1
    for rows, staging in ((62, "plain"), (510, "tma")):
        det.set_tuning(toed.make_params(1.5), rows, staging)
        assert launches(35, 1.5) == 2
        same(35, 1.5)


@pytest.mark.parametrize("group", [2, 31])
def test_lost_copy_in_either_part(toed, group):
    """A ready flag of the first, or the second, of two launches is withheld."""
    _child(f"""
from test_gpu_host_launch import MANY, _many
host = _many(synth)
ref = [r["count"] for r in det.detect_batch([im.cuda() for im in host], sigma=1.5)]
outs = det.alloc_host_outputs(MANY, capacity=200000)
os.environ["TOED_TEST_WITHHOLD_READY"] = "{group}"
os.environ["TOED_TEST_READY_SPINS"] = "20000"
t0 = time.time()
try:
    det.detect_host(host, outs, prm)
    raise SystemExit("no time-out")
except toed.ToedError as e:
    assert e.status == toed.TOED_ERR_TIMEOUT, e
assert time.time() - t0 < 5
got = [int(o["count"].item()) for o in outs]
assert got[:{group}] == ref[:{group}] and got[{group}] == 0, (got, ref)
del os.environ["TOED_TEST_WITHHOLD_READY"], os.environ["TOED_TEST_READY_SPINS"]
det.detect_host(host, outs, prm)
assert [int(o["count"].item()) for o in outs] == ref
print("OK")
""")


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
