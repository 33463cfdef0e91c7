"""The per-pixel passes over interleaved RGB: one result whatever the pixel
count (whole and partial warps' worth, one pixel) and the buffer's alignment
(16 bytes, or an odd multiple of 4).  Exact: a pixel's arithmetic does not
depend on its place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALIB = [0.6722, -0.0635, -0.0963, -0.4287, 1.2460, 0.2028, -0.0908, 0.2162, 0.5668]


def _ops(im):
    return [lambda t: im.exp(t, 0.7), lambda t: im.cfa_coeffs(t, [2.0, 1.0, 1.5]),
            lambda t: im.camera_cst(t, CALIB, im.CS_SRGB), lambda t: im.contrast(t, 1.2), lambda t: im.gamma(t, 2.2),
            lambda t: im.highlight_reconstruction(t, [2.0, 0.9, 1.5]), lambda t: im.sigmoid_tone_map(t),
            lambda t: im.lch(t, im.CS_ACESCG, 1.1, 0.9, 1.0), lambda t: im.cst(t, im.CS_ACESCG, im.CS_OKLCH)]


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 1023, 1024, 5000])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_result_does_not_depend_on_place(gpu, n, offset):
    import torch

    import imops_b200 as im
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.uniform(0.0, 2.0, (8192, 3)).astype(np.float32)).to(gpu)
    for op in _ops(im):
        ref = x.clone()
        op(ref)
        buf = torch.full((3 * n + 8,), -7.0, device=gpu)
        view = buf[offset:offset + 3 * n].view(n, 3)
        view.copy_(x[:n])
        op(view)
        assert torch.equal(view, ref[:n])
        # nothing outside the image is touched
        assert bool((buf[:offset] == -7.0).all()) and bool((buf[offset + 3 * n:] == -7.0).all())


@pytest.mark.parametrize("space", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 129, 5000])
def test_lch_equals_its_three_ops(gpu, space, n):
    """Into Oklch, scaled, and back in one kernel: the bits of the three calls."""
    import torch

    import imops_b200 as im
    x = torch.from_numpy(np.random.default_rng(n).uniform(-0.2, 2.0, (n, 3)).astype(np.float32)).to(gpu)
    one, three = x.clone(), x.clone()
    im.lch(one, space, 1.1, 0.9, 1.05)
    if space != im.CS_OKLCH:
        im.cst(three, space, im.CS_OKLCH)
    im.lch(three, im.CS_OKLCH, 1.1, 0.9, 1.05)
    if space != im.CS_OKLCH:
        im.cst(three, im.CS_OKLCH, space)
    assert torch.equal(one, three)
