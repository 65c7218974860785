"""The FP32 reference-order kernels by features (csrc/wavefront_hybrid.cu) round
as the general ones do: their |z|^2 is spelled out in fused operations, in the
normal stage in another order than elsewhere.  A frame with fast AO takes the
general kernel and one with an AO ray the kernel of its features, so hit, depth,
iteration count, normal and shade of the two are the same bits."""
import pytest

from mandelbulber2_b200 import abi, configs

from .test_gpu_hybrid_kernels import _scene

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "shade")


@pytest.mark.parametrize("name", ["bulb_menger", "bulb_box", "box_menger", "three", "primitive_b", "primitive_x",
                                  "primitive_m", "limits_b", "limits_x", "limits_m", "folds_b", "folds_m"])
def test_lean_equals_general(renderer, name):
    import torch

    renderer.set_scene(_scene(name))
    cam = configs.camera((0.9, -4.2, 1.3), width=211, height=133)
    p = configs.base_params(5, 20.0)
    p.ao_rays, p.ao_fast = 1, 0
    lean = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES)
    p.ao_rays, p.ao_fast = 0, 1
    general = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES)
    for k in NAMES:
        assert torch.equal(lean[k], general[k]), (k, int((lean[k] != general[k]).sum()))
