"""The march jitter's quotient without a division (csrc/jitter.h) is the IEEE quotient for every draw."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_draw(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    csrc = os.path.join(os.path.dirname(HERE), "mandelbulber2_b200", "csrc")
    exe = str(tmp_path / "jitter_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", csrc, os.path.join(HERE, "jitter_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and int(out.stdout) == 0
