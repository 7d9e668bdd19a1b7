"""The decision rounds of the one-CTA-per-trotter sweep, on the host: with the kernel's
own decision functions they end, and take the FP64 outcomes, for ordinary steps and for
infinite, zero, negative, NaN and huge ones, and for couplings of any size."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rounds_end_for_every_step_and_scale(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "rounds")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "sqaod_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "rounds.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
