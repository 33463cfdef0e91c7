"""The adjoint at the sizes where its blur kernels can go wrong: sides just
above the halation radius (both ends of a line in one thread's reach), one off
a tile or a 128-row slab, tall and wide strips, and a radius below 64 (the
general blurs).  Against the FP64 oracle with the relative bar of
tests/test_gpu_adjoint.py (1e-3, entries below 1e-3 of the largest by that)."""
import numpy as np
import pytest

from adjoint_setup import base_vector, perturbed_vector

pytestmark = pytest.mark.gpu

SHAPES = [(66, 66), (67, 130), (129, 97), (257, 66), (66, 1090), (300, 70), (640, 33 + 64)]


def _camera(H, W, seed):
    # camera RGB with highlights above the halation threshold after the white balance
    rng = np.random.default_rng(seed)
    x = rng.random((H, W, 3)) ** 2 * 0.5
    x[H // 3: H // 2, W // 4: W // 2] = 0.9
    x[0, :] = 0.8
    x[:, -1] = 0.7
    return x.astype(np.float32)


@pytest.mark.parametrize("radius", [64, 20])
@pytest.mark.parametrize("H,W", SHAPES)
def test_gradient_on_ragged_frames(oracle_lib, gpu, H, W, radius):
    import torch

    import imops_b200 as im
    oracle = oracle_lib
    x = _camera(H, W, seed=H + W)
    fixed64, fixed = oracle.baseline_params(grain_on=0), im.baseline_film_defaults(grain_on=0)
    fixed64.hal_radius = fixed.hal_radius = radius
    G = oracle.OracleGrad
    tgt = oracle.param_forward(x.astype(np.float64), G.from_vector(perturbed_vector(3)), fixed64).astype(np.float32)
    xd, td = torch.from_numpy(x).to(gpu), torch.from_numpy(tgt).to(gpu)
    p = im.FilmGradParams.from_vector(base_vector())
    v = G.from_vector(base_vector())
    out = im.param_forward(xd, p, fixed).cpu().numpy()
    assert np.abs(out - oracle.param_forward(x.astype(np.float64), v, fixed64)).max() < 1e-4
    scale = 1.0 / x.size
    grad = torch.zeros(25, dtype=torch.float64, device=gpu)
    im.param_backward(xd, p, grad, target=td, loss_scale=scale, fixed=fixed)
    g = grad.cpu().numpy()
    ref = oracle.param_grad(x.astype(np.float64), tgt.astype(np.float64), v, scale, fixed64)
    rel = np.abs(g - ref) / np.maximum(np.abs(ref), 1e-3 * np.abs(ref[:24]).max())
    assert rel.max() < 1e-3, f"worst {int(rel.argmax())}: gpu {g[rel.argmax()]} fp64 {ref[rel.argmax()]}"
    # the same through an upstream gradient
    go = (2.0 * scale * (im.param_forward(xd, p, fixed) - td)).contiguous()
    up = torch.zeros(25, dtype=torch.float64, device=gpu)
    im.param_backward(xd, p, up, g_out=go, fixed=fixed)
    assert torch.allclose(up[:24], grad[:24], rtol=1e-4, atol=1e-6 * float(grad[:24].abs().max()))
