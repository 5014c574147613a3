"""The bounds-checked build over the scan and the edgel kernel: tiles with more
edgels than a chunk, FP64 recomputations, subpixel windows, FP64 lists, and
lists copied to the host band by band.  No check fires and the lists are the
release library's, bit for bit."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import hashlib, json, sys
sys.path.insert(0, {tests!r})
from conftest import load_package
toed = load_package()
import numpy as np, torch
def noise(h, w, dt):
    x = np.clip(np.random.default_rng(h * 7 + w).normal(128, 25, (h, w)), 0, 255)
    return torch.as_tensor(np.rint(x).astype(np.uint8) if dt == "u8" else x.astype(np.float32))
sha = lambda *ts: hashlib.sha1(b"".join(t.contiguous().cpu().numpy().tobytes() for t in ts)).hexdigest()
out = []
for sigma in (0.5, 1.0, 3.0):
    for dt in ("f32", "u8"):
        ims = [noise(h, w, dt) for h, w in ((1, 40), (37, 31), (25, 61), (193, 90), (97, 203), (400, 330))]
        for ori, f64 in ((0, False), (0, True), (1, False), (1, True)):
            det = toed.Detector(0)
            od = toed.TOED_F64 if f64 else toed.TOED_F32
            res = det.detect_batch([im.cuda() for im in ims], sigma=sigma, threshold=0.5, border=1, out_dtype=od, orientation=ori)
            flags = det.flags()
            outs = det.alloc_host_outputs([tuple(im.shape) for im in ims], out_dtype=od, index=True)
            det.detect_host([im.pin_memory() for im in ims], outs, toed.make_params(sigma, 0, 0.5, 1, od, orientation=ori))
            n = [int(o["count"].item()) for o in outs]
            assert n == [r["count"] for r in res]
            dev = sha(*[t for r in res for t in (r["edgels"], r["index"])])
            host = sha(*[t for o, m in zip(outs, n) for t in (o["edgels"][:m], o["index"][:m])])
            out.append([sigma, dt, ori, f64, flags | det.flags(), sum(n), dev, host])
print("RESULT " + json.dumps(out))
"""


def _run(lib_path):
    code = CHILD.format(tests=os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, TOED_LIBRARY=lib_path))
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads([l for l in r.stdout.splitlines() if l.startswith("RESULT ")][-1][7:])


def test_scan_and_edgel_kernel_within_bounds(toed):
    got, ref = _run(toed.build(debug=True)), _run(toed.LIB_PATH)
    assert len(got) == 24 and got == ref
    for sigma, dt, ori, f64, flags, n, dev, host in got:
        assert flags == 0 and n > 2000 and dev == host, (sigma, dt, ori, f64, flags, n)
