"""mbr_kernel_launches counts what was queued: a frame recorded into a graph has
as many kernel nodes, and a batch counts its graph's with every launch.  Frames
by stages cannot be recorded; theirs are stages P, N, S and the finish kernel."""
import ctypes as C

import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import alloc_outputs, outputs_struct

pytestmark = pytest.mark.gpu
NAMES = ("depth", "hit", "normal")


@pytest.mark.parametrize("name,engine", [("box", abi.ENGINE_WAVEFRONT_FP32), ("box", abi.ENGINE_WAVEFRONT_AUTO),
                                         ("box", abi.ENGINE_PLAIN_MIXED), ("box", abi.ENGINE_PLAIN_FP64),
                                         ("hybrid", abi.ENGINE_WAVEFRONT_AUTO), ("gi", abi.ENGINE_WAVEFRONT_FP32),
                                         ("unlit", abi.ENGINE_WAVEFRONT_FP64)])
def test_recorded_kernels(renderer, name, engine):
    import torch

    rt = pytest.importorskip("cuda.bindings.runtime")
    lib = abi.load()
    renderer.set_scene(configs.hybrid_scene() if name in ("hybrid", "gi") else configs.mandelbox_scene(-1.5, 0.5, 20))
    cam = configs.camera((0.3, -5.9, 0.4), width=33, height=21)
    p = configs.base_params(5, 20.0)
    p.ao_rays = 0 if name == "unlit" else 2
    if name == "unlit":
        p.shading_enable = 0
    if name == "gi":
        _, _, p = configs.hybrid_gi_2160p(33, 21, spp=2)
    bufs = alloc_outputs(33 * 21, renderer.device, ("depth", "hit") if name == "unlit" else NAMES)
    renderer.render_into(cam, p, bufs, None, engine)  # the context's scratch, before the recording
    renderer.sync()
    s = torch.cuda.Stream(renderer.device)
    before = lib.mbr_kernel_launches()
    assert int(rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0]) == 0
    renderer.render_into(cam, p, bufs, None, engine, stream=s)
    err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
    assert int(err) == 0
    counted = lib.mbr_kernel_launches() - before
    err, nodes, n = rt.cudaGraphGetNodes(graph, 1000)
    assert int(err) == 0 and n < 1000
    kernel = rt.cudaGraphNodeType.cudaGraphNodeTypeKernel
    assert counted == sum(rt.cudaGraphNodeGetType(x)[1] == kernel for x in nodes[:n])
    rt.cudaGraphDestroy(graph)


def test_staged_frame(renderer):
    lib = abi.load()
    renderer.set_scene(configs.mandelbox_scene(-1.5, 0.5, 20))
    cam = configs.camera((0.3, -5.9, 0.4), width=33, height=21)
    p = configs.base_params(5, 20.0)
    bufs = alloc_outputs(33 * 21, renderer.device, NAMES)
    for ao, kernels in ((4, 4), (0, 1)):
        p.ao_rays = ao
        before = lib.mbr_kernel_launches()
        renderer.render_into(cam, p, bufs, None, abi.ENGINE_PLAIN_FP64)
        assert lib.mbr_kernel_launches() - before == kernels
    renderer.sync()


def test_batch(renderer):
    import torch

    lib = abi.load()
    scenes = (abi.Scene * 2)(configs.mandelbulb_scene(8.0, 40), configs.mandelbox_scene(-1.5, 0.5, 20))
    jobs = (abi.Job * 2)()
    for i in range(2):
        jobs[i].camera = configs.camera((0.3, -5.9, 0.4), width=33, height=21)
        jobs[i].scene_index, jobs[i].pixel_offset = i, i * 33 * 21
    p = configs.base_params(5, 20.0)
    bufs = alloc_outputs(2 * 33 * 21, renderer.device, NAMES)
    o = outputs_struct(bufs, None)
    b = C.c_void_p()
    before = lib.mbr_kernel_launches()
    assert lib.mbr_batch_create(renderer.ctx, scenes, 2, jobs, 2, C.byref(p), C.byref(o), abi.ENGINE_WAVEFRONT_FP32, None,
                                C.byref(b)) == abi.MBR_OK
    try:
        assert lib.mbr_kernel_launches() == before
        s = torch.cuda.current_stream(renderer.device)
        for k in (1, 2):
            assert lib.mbr_batch_launch(b, C.c_void_p(s.cuda_stream)) == abi.MBR_OK
            assert lib.mbr_kernel_launches() == before + k * 12  # two pipelines of six
        renderer.sync()
    finally:
        lib.mbr_batch_destroy(b)
