"""Bands of a plain FP64 frame (row_begin, row_end) take the kernels that the
whole frame takes, so they equal its rows bit for bit: the frames lie above the
size from which frames without AO go through the stages, their bands below."""
import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import alloc_outputs
from mandelbulber2_b200.shard import band_params

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")


@pytest.mark.parametrize("engine", [abi.ENGINE_PLAIN_FP64, abi.ENGINE_PLAIN_FP64_STRICT])
@pytest.mark.parametrize("formula", ["bulb", "box"])
def test_bands_equal_the_frame(renderer, formula, engine):
    import torch

    renderer.set_scene(configs.mandelbulb_scene(8.0, 60) if formula == "bulb" else configs.mandelbox_scene(-1.5, 0.5, 30))
    cam = configs.camera((0.3, -2.9, 0.4) if formula == "bulb" else (0.6, -5.7, 0.8), width=643, height=411)
    p = configs.base_params(5, 20.0)
    whole = renderer.render(cam, p, engine, outputs=NAMES)
    bufs = alloc_outputs(cam.width * cam.height, renderer.device, NAMES)
    for r0, r1 in ((0, 1), (1, 130), (130, 411)):
        renderer.render_into(cam, band_params(p, r0, r1), bufs, None, engine)
    renderer.sync()
    for k in NAMES:
        assert torch.equal(bufs[k], whole[k]), k


@pytest.mark.parametrize("ao_rays,width,height,bands", [
    (0, 512, 300, ((0, 140), (140, 300))), (2, 512, 300, ((0, 140), (140, 300))),
    (1, 1536, 1024, ((0, 60), (60, 1000), (1000, 1024)))])
def test_fp32_mandelbox_bands(renderer, ao_rays, width, height, bands):
    """The FP32 Mandelbox's stage P has three register bounds by the number of pixels: the same bits from each."""
    import torch

    renderer.set_scene(configs.mandelbox_scene(2.2, 0.4, 40))
    cam = configs.camera((3.0, -9.0, 3.0), width=width, height=height)
    p = configs.base_params(5, 30.0)
    p.ao_rays = ao_rays
    whole = renderer.render(cam, p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES)
    bufs = alloc_outputs(cam.width * cam.height, renderer.device, NAMES)
    for r0, r1 in bands:
        renderer.render_into(cam, band_params(p, r0, r1), bufs, None, abi.ENGINE_WAVEFRONT_FP32)
    renderer.sync()
    for k in NAMES:
        assert torch.equal(bufs[k], whole[k]), k
