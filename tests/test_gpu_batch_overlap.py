"""A batch whose jobs write pixels in common: its pipelines run in turn over one
scratch, the FP32 ones by formula kind and then the FP64 ones, so each pixel is
the last pipeline's (jobs apart run side by side)."""
import ctypes as C

import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import STATS_FIELDS, alloc_outputs, outputs_struct, stats_dict

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "rgb8")


@pytest.mark.parametrize("engine", [abi.ENGINE_WAVEFRONT_FP32, abi.ENGINE_WAVEFRONT_AUTO])
def test_the_last_pipeline_stays(renderer, engine):
    import torch

    lib = abi.load()
    # in the order of their pipelines: Mandelbulb, Menger sponge, Mandelbox
    scenes = [configs.mandelbulb_scene(8.0, 60), configs.menger_scene(8), configs.mandelbox_scene(-1.5, 0.5, 30)]
    cams = [configs.camera((0.2, -2.9, 0.4), width=64, height=48), configs.camera((1.2, -3.1, 0.9), width=64, height=48),
            configs.camera((0.6, -5.7, 0.8), width=40, height=25)]
    offsets = [0, 64 * 24, 500]
    n = 64 * 72
    p = configs.base_params(5, 20.0)
    bufs = alloc_outputs(n, renderer.device, NAMES)
    stats = torch.zeros(len(STATS_FIELDS), dtype=torch.int64, device=renderer.device)
    o = outputs_struct(bufs, stats)
    order = (1, 2, 0)  # the order in which the jobs are given does not matter
    jobs = (abi.Job * 3)()
    for i, k in enumerate(order):
        jobs[i].camera, jobs[i].scene_index, jobs[i].pixel_offset = cams[k], k, offsets[k]
    b = C.c_void_p()
    st = lib.mbr_batch_create(renderer.ctx, (abi.Scene * 3)(*scenes), 3, jobs, 3, C.byref(p), C.byref(o), engine, None,
                              C.byref(b))
    assert st == abi.MBR_OK, lib.mbr_last_error_string(renderer.ctx)
    try:
        assert lib.mbr_batch_groups(b, None) == 3
        want = alloc_outputs(n, renderer.device, NAMES)
        for k in range(3):
            renderer.set_scene(scenes[k])
            one = renderer.render(cams[k], p, abi.ENGINE_WAVEFRONT_FP32, outputs=NAMES).buffers
            for name in NAMES:
                want[name][offsets[k]: offsets[k] + cams[k].width * cams[k].height] = one[name]
        s = torch.cuda.current_stream(renderer.device)
        for _ in range(5):
            for v in bufs.values():
                v.zero_()
            stats.zero_()
            assert lib.mbr_batch_launch(b, C.c_void_p(s.cuda_stream)) == abi.MBR_OK
            renderer.sync()
            for name in NAMES:
                assert float((bufs[name] != want[name]).double().mean()) <= 0.001, name
            assert stats_dict(stats)["pixels"] == sum(c.width * c.height for c in cams)
    finally:
        lib.mbr_batch_destroy(b)
