"""Blended sequences, sequences with extensions in GI, and the pseudo-Kleinian DE
function keep their bits on the FP32 wavefront: which products a compiler fuses
in the blend, in the Menger sponge and in that function changes with the code
around them, and with it the iteration counts and 8-bit colours of single pixels.
The digests are of the frames of the kernels as they were before they were split
by features; the orbits use no library function, only IEEE operations."""
import hashlib

import pytest

from mandelbulber2_b200 import abi, configs

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")


def _scene(name):
    if name.endswith("kleinian_de"):
        sc = configs.menger_scene(5) if name.startswith("menger") else configs.mandelbox_scene(-1.5, 0.5, 9)
        sc.delta_de_function = 3  # pseudo-Kleinian
        sc.julia_mode = 1
        sc.julia_c[:] = [0.3, -0.2, 0.1]
        return sc
    sc = configs.mandelbox_scene(-1.5, 0.5, 30)
    sc.hybrid_fractal_enable = 1
    sc.n_fractals = 2
    abi.fractal_defaults(sc.fractal[1], abi.FORMULA_MENGER_SPONGE)
    if name == "box":
        sc.fractal[0].formula_iterations = 3
        sc.fractal[0].formula_weight = 0.8
    elif name == "menger":
        sc.fractal[0].formula_stop_iteration = 2
        sc.fractal[1].formula_weight = 0.7
    else:
        sc.fractal[0].formula_weight = 0.8 if name == "limits" else 1.0
        sc.limits_enabled = 1
        sc.limit_min[:] = [-2.0, -2.0, -2.0]
        sc.limit_max[:] = [2.0, 1.5, 2.0]
    return sc


def digest(renderer, name, kind):
    renderer.set_scene(_scene(name))
    cam = configs.camera((1.8, -5.4, 2.1) if name != "menger_kleinian_de" else (0.7, -2.2, 0.9), width=160, height=120)
    if kind == "gi":
        _, _, p = configs.hybrid_gi_2160p(160, 120, spp=2)
        p.gi_bounces = 3
    else:
        p = configs.base_params(30 if kind == "fast" else 5, 20.0)
        p.ambient_intensity = 0.4
        p.advanced_quality = p.ao_fast = int(kind == "fast")
        p.ao_rays = 2 * int(kind == "ao")
    fr = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES)
    h = hashlib.sha256()
    for k in NAMES:
        if not (kind == "gi" and k == "depth"):
            h.update(fr[k].cpu().numpy().tobytes())
    return h.hexdigest()[:16]


DIGESTS = {
    ("menger_kleinian_de", "ao"): "c03874d6aba3fc7f", ("menger_kleinian_de", "gi"): "e758b48b7fb839d3",
    ("box_kleinian_de", "ao"): "1f6558da8f0581fc",
    ("box", "ao"): "63a0a821407b782a", ("box", "fast"): "a3cf4ad85658f99d", ("box", "gi"): "185b5e58a052f26e",
    ("menger", "ao"): "f6194b13ac09d97f", ("menger", "fast"): "a12cc7497dbf2964", ("menger", "gi"): "f8ff231aef030372",
    ("limits", "ao"): "ab2c26183b5e105d", ("limits", "fast"): "923ed0e032d584f1", ("limits", "gi"): "d541ee2a0a3a6801",
    ("plain_limits", "ao"): "f6d6cb6a925ef78d", ("plain_limits", "fast"): "163b8f7f88a8e17f", ("plain_limits", "gi"): "3e0296767b52a5d4",
}


@pytest.mark.parametrize("name,kind", sorted(DIGESTS))
def test_bits(renderer, name, kind):
    assert digest(renderer, name, kind) == DIGESTS[name, kind]
