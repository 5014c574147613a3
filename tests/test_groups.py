"""The adjoint's group copies stay inside the caller's image and cover what the
windows read (tests/cpp/group_driver.cpp, on the host)."""
import os
import shutil
import subprocess

from conftest import PKG_DIR, ROOT


def test_groups_stay_in_storage(tmp_path):
    exe = str(tmp_path / "groups")
    src = os.path.join(ROOT, "tests", "cpp", "group_driver.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O2", "-I" + os.path.join(PKG_DIR, "csrc"), src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[0]) > 1_000_000, r.stdout
