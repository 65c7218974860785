"""Plain FP64 frames recorded into a CUDA graph: the graph can be cloned, made
a child of another and instantiated twice, as one of kernels and copies can, and
its replay gives the frame (strict engine: bit for bit; with contraction the
depths within 1e-9 and the hits alike)."""
import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import alloc_outputs

pytestmark = pytest.mark.gpu
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")


def _ok(ret):
    assert int(ret[0]) == 0, ret[0]
    return ret[1] if len(ret) == 2 else ret[1:]


@pytest.mark.parametrize("engine", [abi.ENGINE_PLAIN_FP64_STRICT, abi.ENGINE_PLAIN_FP64])
@pytest.mark.parametrize("scene", ["box", "prims"])
def test_recorded_frame(renderer, scene, engine):
    import torch

    rt = pytest.importorskip("cuda.bindings.runtime")
    sc = configs.mandelbox_scene(-1.5, 0.5, 30)
    if scene == "prims":
        sc.n_primitives = 1
        sc.primitive[0] = abi.primitive_defaults(abi.PRIMITIVE_SPHERE)
        sc.primitive[0].position[:] = [1.8, -1.9, 0.4]
    renderer.set_scene(sc)
    cam = configs.camera((0.3, -5.9, 0.4), width=61, height=47)
    p = configs.base_params(5, 20.0)
    p.ao_rays = 4
    direct = renderer.render(cam, p, engine, outputs=NAMES)
    bufs = alloc_outputs(cam.width * cam.height, renderer.device, NAMES)
    s = torch.cuda.Stream(renderer.device)
    h = s.cuda_stream
    _ok(rt.cudaStreamBeginCapture(h, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    renderer.render_into(cam, p, bufs, None, engine, stream=s)
    graph = _ok(rt.cudaStreamEndCapture(h))
    clone = _ok(rt.cudaGraphClone(graph))
    parent = _ok(rt.cudaGraphCreate(0))
    _ok(rt.cudaGraphAddChildGraphNode(parent, None, 0, graph))
    execs = [_ok(rt.cudaGraphInstantiate(g, 0)) for g in (graph, graph, clone, parent)]
    for x in execs:
        for b in bufs.values():
            b.zero_()
        torch.cuda.synchronize()
        _ok(rt.cudaGraphLaunch(x, h) + (None,))
        renderer.sync(s)
        if engine == abi.ENGINE_PLAIN_FP64_STRICT:
            for k in NAMES:
                assert torch.equal(bufs[k], direct[k]), k
        else:
            assert torch.equal(bufs["hit"], direct["hit"])
            hit = direct["hit"].bool()
            rel = ((bufs["depth"] - direct["depth"]) / direct["depth"])[hit].abs()
            assert float(rel.max()) <= 1e-9
    for x in execs:
        _ok(rt.cudaGraphExecDestroy(x) + (None,))
    for g in (parent, clone, graph):
        _ok(rt.cudaGraphDestroy(g) + (None,))
