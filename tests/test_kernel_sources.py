"""Rules of the kernels' sources that no run can show: a wait that gives up
happens on no healthy GPU."""
import glob
import os
import re

from conftest import PKG_DIR


def _kernels():
    """{name: body} of the __global__ functions."""
    out = {}
    for path in sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "*.cu*"))):
        src = open(path).read()
        for m in re.finditer(r"__global__[^;{]*?\b(\w+)\(const __grid_constant__ \w+ \w+\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            out[m.group(1)] = src[m.end():i]
    return out


def test_no_copy_outlives_its_block():
    """A kernel whose wait for a TMA copy gave up waits again, bounded, for what
    is still in flight before it ends, and requests no more copies."""
    kernels = {k: b for k, b in _kernels().items() if "mbar_wait" in b}
    assert set(kernels) == {"toed_detect_kernel", "fin_edgels"}
    for name, body in kernels.items():
        assert body.count("mbar_wait(") == 2, name
        gave_up = body[body.index("mbar_wait("):body.rindex("mbar_wait(")]  # one thread, where the first gave up
        assert "TOED_FLAG_TIMEOUT" in gave_up and "tid == 0" in gave_up and len(gave_up) < 900, name
    assert re.search(r"issued < min\(nbox, upto\) && !dead", kernels["toed_detect_kernel"])


def test_scan_and_edgel_kernel_are_guarded():
    """The bounds-checked build covers every kernel of a detection: the indices
    that data decides -- segments, staged pixels and windows, records, list
    positions, bands -- go through TOED_IN_BOUNDS."""
    kernels = _kernels()
    for name, least in (("toed_detect_kernel", 5), ("fin_scan", 3), ("fin_edgels", 9)):
        assert kernels[name].count("TOED_IN_BOUNDS") >= least, name
    src = open(os.path.join(PKG_DIR, "csrc", "toed_edgels.cuh")).read()
    band = src[src.index("void band_done("):src.index("template <int R, bool QAD>\n__global__")]
    assert band.count("TOED_IN_BOUNDS") >= 3
    # every window handed to a sum is checked against the staged pixels
    body = kernels["fin_edgels"]
    assert len(re.findall(r"const float\* win = ", body)) == body.count("TOED_IN_BOUNDS(staged(win")
