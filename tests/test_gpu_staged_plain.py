"""The plain FP64 engines' staged frames (csrc/staged_plain.cuh): single pixels,
ragged sizes, row bands, the modes whose rules the stages restate, and frames
queued on two streams of one context.  The strict engine is held to the oracle
bit for bit, counters included.  Frames with four AO rays go through the stages
at every size, scenes with a primitive whatever the frame asks for."""
import numpy as np
import pytest

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import STATS_FIELDS, alloc_outputs, stats_dict

pytestmark = pytest.mark.gpu
STRICT = abi.ENGINE_PLAIN_FP64_STRICT
NAMES = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")


def _case(name):
    sc = configs.mandelbox_scene(-1.5, 0.5, 30)
    p = configs.base_params(5, 20.0)
    p.ao_rays = 4
    p.ambient_intensity = 0.4
    if name in ("fast_ao", "fast_ao_of_one", "steps", "unlit"):
        sc.n_primitives = 1
        sc.primitive[0] = abi.primitive_defaults(abi.PRIMITIVE_SPHERE)
        sc.primitive[0].position[:] = [1.8, -1.9, 0.4]
        sc.primitive[0].radius = 0.6
    if name == "interior":
        sc.interior_mode = 1
    elif name == "threshold":
        sc = configs.mandelbox_scene(-1.5, 0.5, 6)
        sc.iteration_threshold_mode = 1
    elif name == "soft":
        p.soft_shadow_cone, p.penetrating = 12.0, 1
    elif name == "fast_ao":
        p.ao_rays, p.ao_fast, p.ao_quality = 0, 1, 3
    elif name == "fast_ao_of_one":
        p.ao_rays, p.ao_fast, p.ao_quality = 0, 1, 1
    elif name == "steps":
        p.max_raymarching_steps = 9
        p.ao_rays = 0
    elif name == "refined":
        p.binary_steps = 30
    elif name == "unlit":
        p.shading_enable = 0
        p.ao_rays = 0
    elif name == "advanced":
        p.advanced_quality = 1
        p.detail_level = 1.6
        p.de_factor = 0.8
    return sc, p


@pytest.mark.parametrize("size", [(1, 1), (9, 5), (67, 41)])
@pytest.mark.parametrize("name", ["plain", "interior", "threshold", "soft", "fast_ao", "fast_ao_of_one", "steps", "refined",
                                  "unlit", "advanced"])
def test_strict_frames(renderer, oracle, name, size):
    sc, p = _case(name)
    cam = configs.camera((1.1, -5.5, 1.7), width=size[0], height=size[1])
    renderer.set_scene(sc)
    o, ost = oracle.render(sc, cam, p)
    fr = renderer.render(cam, p, STRICT, outputs=NAMES)
    for k in NAMES:
        assert np.array_equal(fr[k].cpu().numpy(), o[k]), (name, size, k)
    assert fr.stats == ost


def test_row_band(renderer, oracle):
    import torch

    sc, p = _case("plain")
    cam = configs.camera((1.1, -5.5, 1.7), width=45, height=37)
    whole, _ = oracle.render(sc, cam, p)
    renderer.set_scene(sc)
    p.row_begin, p.row_end = 7, 30
    bufs = alloc_outputs(45 * 37, renderer.device, NAMES)
    for v in bufs.values():
        v.fill_(77)
    stats = torch.zeros(len(STATS_FIELDS), dtype=torch.int64, device=renderer.device)
    renderer.render_into(cam, p, bufs, stats, STRICT)
    renderer.sync()
    assert stats_dict(stats)["pixels"] == 45 * 23
    rows = np.arange(45 * 37) // 45
    inside = (rows >= 7) & (rows < 30)
    for k in NAMES:
        g = bufs[k].cpu().numpy()
        assert np.array_equal(g[inside], whole[k][inside]), k
        assert np.all(g[~inside] == 77), k


def test_two_streams(renderer):
    """Frames of different size queued on two streams of one context, in turn: each has its own scratch."""
    import torch

    sc, p = _case("plain")
    renderer.set_scene(sc)
    cams = [configs.camera((1.1, -5.5, 1.7), width=w, height=h) for w, h in ((211, 97), (64, 203))]
    alone = [renderer.render(c, p, STRICT, outputs=NAMES).buffers for c in cams]
    streams = [torch.cuda.Stream(renderer.device) for _ in cams]
    bufs = [alloc_outputs(c.width * c.height, renderer.device, NAMES) for c in cams]
    torch.cuda.synchronize()
    for _ in range(4):
        for c, s, b in zip(cams, streams, bufs):
            renderer.render_into(c, p, b, None, STRICT, stream=s)
    for s in streams:
        renderer.sync(s)
    for a, b in zip(alone, bufs):
        for k in NAMES:
            assert torch.equal(a[k], b[k]), k
