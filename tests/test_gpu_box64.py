"""The FP64 wavefront's Mandelbox iteration (csrc/wavefront.cuh, Prec64) where
its folds branch: a tiny minimum radius (a large sphere-fold factor),
radii that lie close together, a positive scale, a Julia constant, c left out.
Held to the FP64 wavefront's bars against the oracle: hits and iteration counts
identical on >= 99.9 % of the pixels, depth within 1e-9 on >= 99.9 % of the
common hits."""
import pytest

from mandelbulber2_b200 import abi, configs

from .parity import compare

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "ao", "rgb8")


def _scene(name):
    sc = configs.mandelbox_scene(-1.5, 0.5, 50)
    f = sc.fractal[0]
    if name == "tiny_min_radius":
        f.mandelbox_folding_min_radius = 1e-3
    elif name == "close_radii":
        f.mandelbox_folding_min_radius = 0.999
    elif name == "positive_scale":
        sc = configs.mandelbox_scene(2.3, 0.35, 30)
    elif name == "julia":
        sc = configs.mandelbox_scene(2.0, 0.5, 30)
        sc.julia_mode = 1
        sc.julia_c[:] = [0.4, -0.3, 0.2]
        sc.fractal_constant_factor[:] = [1.1, 0.9, 1.3]
    elif name == "no_c":
        f.dont_add_c_constant = 1
        sc.formula_maxiter = 12
    return sc


@pytest.mark.parametrize("name", ["tiny_min_radius", "close_radii", "positive_scale", "julia", "no_c"])
def test_box_folds(renderer, oracle, name):
    sc, cam, p = configs.mandelbox_1080p("A", 95, 53, ao_rays=2)
    sc = _scene(name)
    renderer.set_scene(sc)
    fr = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP64, outputs=NAMES)
    o, _ = oracle.render(sc, cam, p)
    m = compare({k: v.cpu().numpy() for k, v in fr.buffers.items()}, o)
    print(name, float(o["hit"].mean()), m)
    assert m["hit_mismatch"] <= 0.001, m
    if o["hit"].any():
        assert m["hit_iters_match"] >= 0.999, m
        assert m["depth_rel_le_1e-9"] >= 0.999, m
