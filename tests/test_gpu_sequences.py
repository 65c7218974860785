"""Hybrid sequences through the kernels that step an orbit pass by pass
(orbit_pass, csrc/de_core.cuh): the distance queries' refilling kernel and the
staged plain FP64 frames, and the staged frames of blended sequences, whose
estimates are taken whole.  Mandelbox and Menger slots round as the oracle does,
so the strict engine equals it bit for bit, counters included: start and stop
iterations, the slot the sequence repeats from, slots that do not check the
bailout, a Julia constant, an unused weighted slot, points that are not finite.
The engine with contraction is held to the FP64 bars (hits and iteration counts
identical on >= 99.9 % of the pixels, depth within 1e-9 on >= 99.9 %)."""
import numpy as np
import pytest

from mandelbulber2_b200 import abi, configs

from .parity import compare

pytestmark = pytest.mark.gpu
STRICT = abi.ENGINE_PLAIN_FP64_STRICT
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")
BOX, MENGER = abi.FORMULA_MANDELBOX, abi.FORMULA_MENGER_SPONGE


def _sequence(name):
    sc = configs.mandelbox_scene(-1.5, 0.5, 17)
    sc.hybrid_fractal_enable = 1
    sc.n_fractals = 3
    sc.fractal[0].formula_iterations = 2
    abi.fractal_defaults(sc.fractal[1], MENGER)
    abi.fractal_defaults(sc.fractal[2], BOX)
    sc.fractal[2].mandelbox_scale = 2.1
    sc.fractal[2].mandelbox_folding_min_radius = 0.4
    if name == "ranges":
        sc.fractal[0].formula_stop_iteration = 5
        sc.fractal[1].formula_start_iteration = 2
        sc.fractal[2].formula_start_iteration = 4
        sc.fractal[2].formula_iterations = 3
        sc.repeat_from = 2
    elif name == "unchecked":
        sc.fractal[0].check_for_bailout = 0
        sc.fractal[2].check_for_bailout = 0
        sc.use_default_bailout = 0
        sc.bailout = 7.5
    elif name == "julia":
        sc.julia_mode = 1
        sc.julia_c[:] = [0.3, -0.2, 0.1]
        sc.fractal[1].dont_add_c_constant = 0
    elif name == "unused_weight":  # never live, so it does not blend
        sc.fractal[2].formula_start_iteration = 9000
        sc.fractal[2].formula_stop_iteration = 9000
        sc.fractal[2].formula_weight = 0.5
    elif name == "blended":
        sc.fractal[1].formula_weight = 0.8
    return sc


SEQUENCES = ["plain", "ranges", "unchecked", "julia", "unused_weight", "blended"]


@pytest.mark.parametrize("name", SEQUENCES + ["menger"])
def test_distances(renderer, oracle, name):
    """310003 points: on 148 SMs every warp of either kernel's largest grid takes a second group."""
    import torch

    sc = configs.menger_scene(9) if name == "menger" else _sequence(name)
    renderer.set_scene(sc)
    pts = np.random.default_rng(17).uniform(-2.5, 2.5, size=(310003, 3))
    for k, special in enumerate(([0.0, 0.0, 0.0], [np.inf, 0.0, 1.0], [np.nan, 1.0, 2.0], [1e200, 0.0, 0.0],
                                 [-1.0, 1.0, -1.0])):
        pts[37 * (k + 1)] = pts[310002 - 41 * k] = special
    for n in (1, 33, 310003):
        for normal_mode in (False, True):
            d, it = renderer.distance(torch.from_numpy(pts[:n]), 1e-3, normal_mode, STRICT)
            od, oit = oracle.distance(sc, pts[:n], 1e-3, normal_mode)
            assert np.array_equal(it.cpu().numpy(), oit), n
            assert np.array_equal(d.cpu().numpy(), od, equal_nan=True), n


@pytest.mark.parametrize("size", [(1, 1), (61, 37)])
@pytest.mark.parametrize("name", SEQUENCES)
def test_staged_frames(renderer, oracle, name, size):
    sc = _sequence(name)
    cam = configs.camera((1.0, -4.6, 1.4), width=size[0], height=size[1])
    p = configs.base_params(5, 20.0)
    p.ao_rays = 4
    p.ambient_intensity = 0.4
    renderer.set_scene(sc)
    o, ost = oracle.render(sc, cam, p)
    fr = renderer.render(cam, p, STRICT, outputs=NAMES)
    for k in NAMES:
        assert np.array_equal(fr[k].cpu().numpy(), o[k]), k
    assert fr.stats == ost
    if size != (1, 1):
        fma = renderer.render(cam, p, abi.ENGINE_PLAIN_FP64, outputs=NAMES)
        m = compare({k: v.cpu().numpy() for k, v in fma.buffers.items()}, o)
        print(name, m)
        assert o["hit"].any()
        assert m["hit_iters_match"] >= 0.999 and m["depth_rel_le_1e-9"] >= 0.999, m
