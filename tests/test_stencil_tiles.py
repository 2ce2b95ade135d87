"""The order in which the TMA stencil kernels take their tiles, checked on the CPU
(tests/c/st_tiles_check.cpp)."""
import os
import subprocess

from blopex_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_tile_once(tmp_path):
    exe = str(tmp_path / "st_tiles_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", build.CSRC, os.path.join(ROOT, "tests", "c", "st_tiles_check.cpp"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
