"""A sequence without a live slot at iteration 0: its table is one entry long
and names slot 0, which may be empty.  Every pass then leaves the point where
it is, and the distance is that of the unit sphere for a linear DE offset of 1:
(|p| - 1) / 1.  The engines that choose a kernel by the formulas of the scene
have to see the empty slot."""
import numpy as np
import pytest

from mandelbulber2_b200 import abi, configs

from .parity import compare

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "ao", "rgb8")


def _scene(late):
    sc = configs.menger_scene(6)
    sc.hybrid_fractal_enable = 1
    sc.linear_de_offset = 1.0
    sc.n_fractals = 1 + len(late)
    sc.fractal[0].formula = abi.FORMULA_NONE
    for k, formula in enumerate(late):
        abi.fractal_defaults(sc.fractal[1 + k], formula)
        sc.fractal[1 + k].formula_start_iteration = 1
    return sc


LATE = [(abi.FORMULA_MENGER_SPONGE,), (abi.FORMULA_MANDELBOX, abi.FORMULA_MENGER_SPONGE),
        (abi.FORMULA_MENGER_SPONGE, abi.FORMULA_MANDELBOX, abi.FORMULA_MENGER_SPONGE)]


@pytest.mark.parametrize("late", LATE)
def test_distances(renderer, late):
    import torch

    renderer.set_scene(_scene(late))
    pts = np.random.default_rng(5).uniform(-3.0, 3.0, size=(4099, 3))
    want = np.clip(np.sqrt((pts * pts).sum(1)) - 1.0, 0.0, 10.0)
    for engine, tol in ((abi.ENGINE_PLAIN_FP64_STRICT, 1e-14), (abi.ENGINE_PLAIN_FP64, 1e-14), (abi.ENGINE_PLAIN_MIXED, 2e-6)):
        d, _ = renderer.distance(torch.from_numpy(pts), 1e-3, False, engine)
        assert np.abs(d.cpu().numpy() - want).max() <= tol, engine


@pytest.mark.parametrize("engine", [abi.ENGINE_PLAIN_FP64, abi.ENGINE_WAVEFRONT_FP32, abi.ENGINE_WAVEFRONT_AUTO])
@pytest.mark.parametrize("late", LATE)
def test_frames(renderer, late, engine):
    """Held to the FP32 bars against the strict FP64 engine's frame."""
    renderer.set_scene(_scene(late))
    cam = configs.camera((0.9, -2.6, 0.8), width=67, height=41)
    p = configs.base_params(5, 20.0)
    p.ao_rays = 4
    ref = renderer.render(cam, p, abi.ENGINE_PLAIN_FP64_STRICT, outputs=NAMES)
    fr = renderer.render(cam, p, engine, outputs=NAMES)
    a, b = ({k: v.cpu().numpy() for k, v in f.buffers.items()} for f in (fr, ref))
    m = compare(a, b)
    print(m)
    assert b["hit"].mean() > 0.2
    assert m["hit_mismatch"] <= 0.005, m
    assert m["depth_rel_median"] <= 1e-4, m
    assert abs(fr.stats["de_evals"] - ref.stats["de_evals"]) <= 0.05 * ref.stats["de_evals"]
