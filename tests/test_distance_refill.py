"""CalculateDistance over uneven points: the kernel that refills the lanes of
finished orbits (csrc/plain_kernel.cuh) and its bailout on |z|^2
(csrc/bailout.h).  Both leave every operation of an orbit as it was, so the
comparisons are for equality."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from mandelbulber2_b200 import abi, configs

HERE = os.path.dirname(os.path.abspath(__file__))


def test_bailout_on_the_square(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    csrc = os.path.join(os.path.dirname(HERE), "mandelbulber2_b200", "csrc")
    exe = str(tmp_path / "bailout_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", csrc, os.path.join(HERE, "bailout_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    bad, checked = map(int, out.stdout.split())
    assert checked > 1_000_000
    assert bad == 0 and out.returncode == 0


def _scenes():
    box = configs.mandelbox_scene(-1.5, 0.5, 50)
    julia = configs.mandelbox_scene(2.0, 0.4, 20)
    julia.julia_mode = 1
    julia.julia_c[:] = [0.3, -0.2, 0.1]
    julia.min_n = 4
    julia.use_default_bailout = 0
    julia.bailout = 7.3
    inside = configs.menger_scene(6)
    inside.interior_mode = 1
    threshold = configs.mandelbox_scene(-1.5, 0.5, 7)
    threshold.iteration_threshold_mode = 1
    weightless = configs.menger_scene(5)
    weightless.fractal[0].formula_weight = 0.0
    mixed = configs.mandelbox_scene(-1.5, 0.5, 17)
    mixed.hybrid_fractal_enable = 1
    mixed.n_fractals = 2
    mixed.fractal[0].formula_iterations = 2
    mixed.fractal[0].formula_weight = 0.8
    abi.fractal_defaults(mixed.fractal[1], abi.FORMULA_MENGER_SPONGE)
    return {"box": box, "julia": julia, "menger": configs.menger_scene(12), "interior": inside,
            "threshold": threshold, "weightless": weightless, "hybrid": mixed}


def _points(n):
    pts = np.random.default_rng(11).uniform(-2.5, 2.5, size=(n, 3))
    for k, special in enumerate(([0.0, 0.0, 0.0], [np.inf, 0.0, 1.0], [np.nan, 1.0, 2.0], [1e200, 0.0, 0.0],
                                 [-1.0, 1.0, -1.0])):
        if n > 40 * (k + 1):
            pts[37 * (k + 1)] = special
    return pts


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(_scenes()) if os.path.exists(abi.LIB_PATH) else [])
def test_strict_equals_the_oracle(renderer, oracle, name):
    import torch

    sc = _scenes()[name]
    renderer.set_scene(sc)
    for n in (1, 31, 33, 4099, 150001):  # 150001 points: more groups than resident warps
        pts = _points(n)
        for normal_mode in (False, True):
            d, it = renderer.distance(torch.from_numpy(pts), 1e-3, normal_mode, abi.ENGINE_PLAIN_FP64_STRICT)
            od, oit = oracle.distance(sc, pts, 1e-3, normal_mode)
            assert np.array_equal(it.cpu().numpy(), oit), (name, n)
            assert np.array_equal(d.cpu().numpy(), od, equal_nan=True), (name, n)


@pytest.mark.gpu
@pytest.mark.parametrize("engine", [abi.ENGINE_PLAIN_FP64, abi.ENGINE_PLAIN_FP64_STRICT, abi.ENGINE_PLAIN_MIXED])
def test_a_point_does_not_depend_on_its_neighbours(renderer, engine):
    """The Mandelbulb (250 iterations inside, a few outside): one call equals calls of a warp's points and fewer."""
    import torch

    renderer.set_scene(configs.mandelbulb_scene(8.0, 250))
    pts = torch.from_numpy(np.random.default_rng(12).uniform(-1.2, 1.2, size=(90001, 3)))
    d, it = renderer.distance(pts, 1e-3, False, engine)
    for a, b in ((0, 1), (5, 36), (100, 132), (4000, 4131), (80000, 90001)):
        dd, ii = renderer.distance(pts[a:b], 1e-3, False, engine)
        assert torch.equal(dd, d[a:b]) and torch.equal(ii, it[a:b]), (a, b)
