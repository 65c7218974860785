"""The adjoint's kernels (csrc/adjoint.cu): eight lanes per hit, and one thread
per pixel for Mandelbox images of 16384 pixels and more.  On both sides of that
line and at ragged sizes the gradient equals the sum of the oracle's per-pixel
forward-mode gradients.  Bar: 1e-6, that of tests/test_gpu_adjoint.py, of the
sum of the magnitudes of its terms."""
import numpy as np
import pytest
import torch

from mandelbulber2_b200 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,size", [("mandelbulb", (1, 1)), ("mandelbulb", (7, 5)), ("mandelbulb", (61, 67)),
                                       ("mandelbulb", (131, 127)), ("mandelbox", (3, 2)), ("mandelbox", (127, 129)),
                                       ("mandelbox", (128, 128)), ("mandelbox", (149, 113))])
@pytest.mark.parametrize("weights", ["both", "depth", "shade", "sparse"])
def test_gradient_is_the_sum_of_the_pixels(renderer, oracle, kind, size, weights):
    sc, cam, p = configs.adjoint_256(kind, *size)
    renderer.set_scene(sc)
    o, _ = oracle.render(sc, cam, p)
    n = size[0] * size[1]
    rng = np.random.default_rng(n)
    wt, ws = rng.uniform(-1.0, 1.0, n).astype(np.float32), rng.uniform(-1.0, 1.0, n).astype(np.float32)
    if weights == "sparse":
        wt[rng.uniform(size=n) < 0.9] = 0.0
        ws[rng.uniform(size=n) < 0.7] = 0.0
    dev = renderer.device
    depth, hit = torch.from_numpy(o["depth"]).to(dev), torch.from_numpy(o["hit"]).to(dev)
    dlt = None if weights == "shade" else torch.from_numpy(wt).to(dev)
    dls = None if weights == "depth" else torch.from_numpy(ws).to(dev)
    g = renderer.adjoint(cam, p, depth, hit, dlt, dls, abi.ENGINE_PLAIN_FP64).cpu().numpy()
    dt, ds, _ = oracle.pixel_gradients(sc, cam, p, o["depth"], o["hit"])
    terms = (0.0 if dlt is None else wt.astype(np.float64)[:, None] * dt) + \
            (0.0 if dls is None else ws.astype(np.float64)[:, None] * ds)
    want, size_of = terms.sum(0), np.abs(terms).sum(0)
    for k in range(abi.GRAD_COUNT - 1):
        assert abs(g[k] - want[k]) <= 1e-6 * size_of[k] + 1e-300, (k, g[k], want[k], size_of[k])
