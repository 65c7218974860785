"""The FP32 wavefront's reference-order kernels by what a scene needs
(csrc/wavefront_hybrid.cu): sequences of every pair and of all three formulas,
single formulas with primitives, limit box or folds, and the general kernels
(a blended slot, fast AO).  Held to the FP32 bars against the oracle: hit
mismatch <= 0.5 %, median relative depth error <= 1e-4, DE counts within 5 %.
(The folded Mandelbox is left out: it encloses this camera, and where every
pixel hits at depth 0 an FP32 depth says nothing.)"""
import pytest

from mandelbulber2_b200 import abi, configs

from .parity import compare

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "ao", "rgb8")
BULB, BOX, MENGER = abi.FORMULA_MANDELBULB, abi.FORMULA_MANDELBOX, abi.FORMULA_MENGER_SPONGE


def _sequence(*formulas):
    sc = abi.scene_defaults(formulas[0])
    sc.formula_maxiter = 14
    sc.hybrid_fractal_enable = 1
    sc.n_fractals = len(formulas)
    for k, f in enumerate(formulas):
        abi.fractal_defaults(sc.fractal[k], f)
        sc.fractal[k].formula_iterations = 2
        sc.fractal[k].bulb_power = 8.0
        sc.fractal[k].mandelbox_scale = -1.5
    return sc


def _scene(name):
    if name == "bulb_menger":
        return _sequence(BULB, MENGER)
    if name == "bulb_box":
        return _sequence(BULB, BOX)
    if name == "box_menger":
        return _sequence(BOX, MENGER)
    if name == "three":
        return _sequence(BOX, BULB, MENGER)
    if name == "blend":
        sc = _sequence(BULB, MENGER)
        sc.fractal[0].formula_weight = 0.8
        return sc
    sc = {"b": configs.mandelbulb_scene(8.0, 40), "x": configs.mandelbox_scene(-1.6, 0.5, 30),
          "m": configs.menger_scene(8)}[name[-1]]
    if name.startswith("primitive"):
        sc.n_primitives = 1
        sc.primitive[0] = abi.primitive_defaults(abi.PRIMITIVE_SPHERE)
        sc.primitive[0].position[:] = [1.4, -0.3, 0.6]
        sc.primitive[0].radius = 0.5
    elif name.startswith("limits"):
        sc.limits_enabled = 1
        sc.limit_min[:] = [-1.1, -5.0, -5.0]
        sc.limit_max[:] = [5.0, 5.0, 0.7]
    else:
        sc.box_folding = sc.spherical_folding = 1
    return sc


@pytest.mark.parametrize("name", ["bulb_menger", "bulb_box", "box_menger", "three", "blend", "primitive_b", "primitive_x",
                                  "primitive_m", "limits_b", "limits_x", "limits_m", "folds_b", "folds_m"])
@pytest.mark.parametrize("fast", [0, 1])
def test_reference_order_kernels(renderer, oracle, name, fast):
    sc = _scene(name)
    cam = configs.camera((0.9, -4.2, 1.3), width=67, height=41)
    p = configs.base_params(5, 20.0)
    p.ao_rays = 0 if fast else 2
    p.ao_fast = fast
    renderer.set_scene(sc)
    o, ost = oracle.render(sc, cam, p)
    fr = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES)
    m = compare({k: v.cpu().numpy() for k, v in fr.buffers.items()}, o)
    print(name, float(o["hit"].mean()), m)
    assert m["hit_mismatch"] <= 0.005, m
    if o["hit"].any():
        assert m["depth_rel_median"] <= 1e-4, m
    assert abs(fr.stats["de_evals"] - ost["de_evals"]) <= 0.05 * ost["de_evals"]
