"""Twiddle grids of the complex128 four-step passes are formed from an eighth of
the circle's fixed-point words; every word equals the direct conversion's."""
import json
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "fixed_circle.cu")


def test_fixed_circle_words(tmp_path):
    from qusim_gb300 import build
    exe = str(tmp_path / "fixed_circle")
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + [SRC, "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=120).stdout
    assert json.loads(out) == {str(n): 0 for n in (8, 16, 24, 4096, 6000, 131072)}
