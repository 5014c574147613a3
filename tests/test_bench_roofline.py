"""bench.py's HBM roofline: bytes and time are those of the same three kernels."""
import os
import re

from conftest import ROOT


def test_bytes_and_time_are_the_steps():
    import bench
    r = bench.hbm_roofline(79_422_768, 2_422_903, 64, 1.691, 6689.5)
    # 4 bytes a pixel, 16 an edgel, 4 an image: 356.5 MB in 1.691 ms
    assert r["achieved"] == round((79_422_768 * 4 + 2_422_903 * 16 + 256) / 1.691e-3 / 1e9, 2) == 210.8
    assert r["frac"] == round(r["achieved"] / 6689.5, 5) or abs(r["frac"] - r["achieved"] / 6689.5) < 1e-5
    src = open(os.path.join(ROOT, "bench.py")).read()
    assert "hbm_roofline(npx, n_edgels, len(images), ms, hbm_peak)" in src  # a graph replay's time


def test_traffic_is_the_sum_of_the_kernels():
    import bench
    path = os.path.join(ROOT, "profiles", "toed_detect_kernel__uneven_batch64_sigma1.5.traffic.txt")
    text = open(path).read()
    rows = re.findall(r"^# (toed_detect_kernel|fin_scan|fin_edgels):\s+read\s+([\d,]+) written\s+([\d,]+)", text, re.M)
    assert [r[0] for r in rows] == ["toed_detect_kernel", "fin_scan", "fin_edgels"]
    total = sum(int(x.replace(",", "")) for r in rows for x in r[1:])
    assert f"dram_bytes_per_step {total}" in text
    px = int(re.search(r"^pixels (\d+)", text, re.M).group(1))
    assert bench.hbm_roofline(px, 0, 0, 1.0, 1.0)["traffic"] == total
