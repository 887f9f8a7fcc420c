"""Launch set-up kept per device (tests/cxx/per_device.cpp, with a stand-in for the CUDA runtime), and no launcher of
the kernels with opt-in shared memory keeps it in a plain static."""
import os
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
KERNELS = ROOT / "tandem_b200/csrc/kernels"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))


def test_per_device(tmp_path):
    exe = tmp_path / "per_device"
    cmd = ["g++", "-std=c++17", "-O1", "-pthread", "-Wall", "-Wextra", "-Werror", "-I", str(ROOT / "tandem_b200/csrc"),
           "-isystem", str(CUDA / "include"), str(ROOT / "tests/cxx/per_device.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["0"], r.stdout + r.stderr


def test_launchers_keep_no_plain_static():
    for name in ("bjacobi.cu", "apply_warp.cu", "apply_warp32_impl.cuh", "warp_plan.hpp"):
        text = (KERNELS / name).read_text()
        assert not re.search(r"\bstatic (?!PerDevice)(bool|int|size_t|const)\b(?! ?\w*\()", text), name
