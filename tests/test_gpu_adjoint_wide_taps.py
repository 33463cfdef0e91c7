"""The adjoint with a halation almost as flat as its window is wide (sigma near
the radius): every tap weighs about 1/(2R + 1), so that one left out, doubled
or at the wrong place moves the halation's share by a hundredth or more; and
against a target well below the output, so that the residuals have one sign
and no gradient is a difference of nearly equal sums.

Bar 5e-5 relative (entries below 1e-2 of the largest by that): a pixel's f32
chain (scan, curves, blurs of 129 taps) is good to about 1e-6, the sums are
in f64, and the sums of both signs (sigma's, the matrix's) lose a digit."""
import numpy as np
import pytest

from adjoint_setup import base_vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,sigma", [(64, 60.0), (20, 18.0)])
@pytest.mark.parametrize("H,W", [(67, 66), (129, 140), (131, 1090), (300, 200)])
def test_gradient_with_flat_taps(oracle_lib, gpu, H, W, radius, sigma):
    import torch

    import imops_b200 as im
    oracle = oracle_lib
    rng = np.random.default_rng(H + W + radius)
    x = (0.02 + rng.random((H, W, 3)) ** 2 * 0.9).astype(np.float32)
    fixed64, fixed = oracle.baseline_params(grain_on=0), im.baseline_film_defaults(grain_on=0)
    fixed64.hal_radius = fixed.hal_radius = radius
    fixed64.hal_threshold = fixed.hal_threshold = 0.1
    v = base_vector()
    v[22], v[23] = 0.5, sigma  # halation strength and sigma
    theta64, theta = oracle.OracleGrad.from_vector(v), im.FilmGradParams.from_vector(v)
    ref_out = oracle.param_forward(x.astype(np.float64), theta64, fixed64)
    tgt = (ref_out - 0.1 - 0.2 * rng.random((H, W, 3))).astype(np.float32)
    scale = 1.0 / x.size
    grad = torch.zeros(25, dtype=torch.float64, device=gpu)
    im.param_backward(torch.from_numpy(x).to(gpu), theta, grad, target=torch.from_numpy(tgt).to(gpu), loss_scale=scale,
                      fixed=fixed)
    g = grad.cpu().numpy()
    ref = oracle.param_grad(x.astype(np.float64), tgt.astype(np.float64), theta64, scale, fixed64)
    rel = np.abs(g - ref) / np.maximum(np.abs(ref), 1e-2 * np.abs(ref[:24]).max())
    assert rel.max() < 5e-5, f"worst {int(rel.argmax())}: gpu {g[rel.argmax()]} fp64 {ref[rel.argmax()]}"
