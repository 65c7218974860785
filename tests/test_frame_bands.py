"""Plain FP64 frames whose scratch would pass the limit are rendered in bands of
rows over one bounded scratch (csrc/frame_bands.h)."""
import os
import shutil
import subprocess

import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import STATS_FIELDS, alloc_outputs, stats_dict
from mandelbulber2_b200.shard import band_params

HERE = os.path.dirname(os.path.abspath(__file__))


def test_choice_of_the_band(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    csrc = os.path.join(os.path.dirname(HERE), "mandelbulber2_b200", "csrc")
    exe = str(tmp_path / "frame_bands_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", csrc, os.path.join(HERE, "frame_bands_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    bad, checked = map(int, out.stdout.split())
    assert checked > 1000
    assert bad == 0 and out.returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("engine", [abi.ENGINE_PLAIN_FP64, abi.ENGINE_PLAIN_FP64_STRICT])
def test_a_large_frame_equals_its_parts(renderer, engine):
    """A distant Mandelbulb with 64 AO rays whose whole scratch would be 25 GB: one call equals calls of its parts."""
    import torch

    renderer.set_scene(configs.mandelbulb_scene(8.0, 30))
    cam = configs.camera((5.0, -59.0, 6.0), width=8192, height=5120)
    p = configs.base_params(5, 100.0)
    p.ao_rays = 64
    names = ("depth", "iters", "hit", "ao")
    n = cam.width * cam.height
    frames, counts = [], []
    for parts in (((0, 5120),), ((0, 2500), (2500, 2571), (2571, 5120))):
        bufs = alloc_outputs(n, renderer.device, names)
        stats = torch.zeros(len(STATS_FIELDS), dtype=torch.int64, device=renderer.device)
        for r0, r1 in parts:
            renderer.render_into(cam, band_params(p, r0, r1), bufs, stats, engine)
        renderer.sync()
        frames.append(bufs)
        counts.append(stats_dict(stats))
    assert 20000 < int(frames[0]["hit"].sum()) < n // 4
    for k in names:
        assert torch.equal(frames[0][k], frames[1][k]), k
    assert counts[0] == counts[1] and counts[0]["pixels"] == n
