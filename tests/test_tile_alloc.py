"""Filling the apply's geometry tiles (in parallel, at upload) allocates nothing: tests/cxx/tile_alloc.cpp, the
product's host sources with a counting operator new."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_no_allocation_in_the_parallel_region(tmp_path):
    exe = tmp_path / "tile_alloc"
    host = ROOT / "tandem_b200/csrc/host"
    cmd = ["g++", "-std=c++17", "-O1", "-fopenmp", "-I", str(ROOT / "tandem_b200/csrc"), "-I", str(ROOT / "include"),
           str(ROOT / "tests/cxx/tile_alloc.cpp"), *[str(host / f) for f in ("refelem.cpp", "setup.cpp", "warp_tables.cpp")],
           "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["0"], r.stdout + r.stderr
