"""Where plain FP64 frames change from the per-pixel kernels to the stages
(staged_plain_takes, csrc/staged_plain.cuh), on either side of each line: trees
by their AO rays, the Menger sponge with a primitive and a sequence in a limit
box by AO and by size, the delta DE never, frames of the specialised formulas by
AO and by size.  The strict engine equals the
oracle bit for bit on both sides, counters included."""
import numpy as np
import pytest

from mandelbulber2_b200 import abi, configs
from tests.golden.pipeline_cases import _trees

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")


def _menger_with_sphere():
    sc = configs.menger_scene(8)
    sc.n_primitives = 1
    sc.primitive[0] = abi.primitive_defaults(abi.PRIMITIVE_SPHERE)
    sc.primitive[0].position[:] = [1.2, -0.9, 0.4]
    sc.primitive[0].radius = 0.6
    return sc


def _limits_hybrid():
    sc = configs.mandelbox_scene(-1.5, 0.5, 12)
    sc.hybrid_fractal_enable = 1
    sc.n_fractals = 2
    abi.fractal_defaults(sc.fractal[1], abi.FORMULA_MENGER_SPONGE)
    sc.limits_enabled = 1
    sc.limit_min[:] = [-3.0, -3.0, -3.0]
    sc.limit_max[:] = [3.0, 3.0, 0.9]
    return sc


def _delta():
    sc = configs.mandelbox_scene(-1.5, 0.5, 10)
    sc.delta_de_method = abi.DE_METHOD_FORCE_DELTA
    return sc


CASES = [("tree", 40, 30, 3, 0), ("tree", 40, 30, 4, 0), ("tree", 40, 30, 0, 1), ("menger_sphere", 160, 119, 0, 0),
         ("menger_sphere", 160, 120, 0, 0), ("menger_sphere", 31, 17, 1, 0), ("menger_sphere", 31, 17, 0, 1),
         ("menger_sphere", 31, 17, 4, 0), ("limits_hybrid", 160, 119, 1, 0), ("limits_hybrid", 160, 120, 1, 0),
         ("delta", 33, 21, 4, 0), ("delta", 33, 21, 0, 0), ("box", 33, 21, 3, 0), ("box", 33, 21, 4, 0), ("box", 512, 511, 0, 0), ("box", 512, 512, 0, 0)]


@pytest.mark.parametrize("name,width,height,ao,fast", CASES)
def test_both_sides(renderer, oracle, name, width, height, ao, fast):
    sc = {"tree": lambda: _trees()["tree_disabled_branch"], "menger_sphere": _menger_with_sphere,
          "limits_hybrid": _limits_hybrid, "delta": _delta,
          "box": lambda: configs.mandelbox_scene(-1.5, 0.5, 12)}[name]()
    cam = configs.camera({"tree": (0.0, -8.0, 1.0), "menger_sphere": (1.2, -3.6, 1.4)}.get(name, (1.1, -5.5, 1.7)),
                         width=width, height=height)
    p = configs.base_params(5, 20.0)
    p.ao_rays, p.ao_fast, p.ambient_intensity = ao, fast, 0.4
    renderer.set_scene(sc)
    o, ost = oracle.render(sc, cam, p)
    fr = renderer.render(cam, p, abi.ENGINE_PLAIN_FP64_STRICT, outputs=NAMES)
    assert o["hit"].any()
    for k in NAMES:
        assert np.array_equal(fr[k].cpu().numpy(), o[k]), k
    assert fr.stats == ost
