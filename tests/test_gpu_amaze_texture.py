"""AMaZE on frames full of texture near the sampling limit, where most tiles'
Nyquist boxes hold voted sites in every density: bit for bit the CPU oracle,
as everywhere (the area sums' order decides bits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _texture(H, W, share, seed):
    """Stripes of two pixels' period in patches that cover `share` of the
    frame, faint noise on all of it."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:H, 0:W]
    stripes = 0.5 + 0.4 * np.where(rng.random() < 0.5, np.cos(np.pi * x * 0.98 + 0.3), np.cos(np.pi * y * 0.98 + 0.3))
    patch = rng.random(((H + 12) // 13, (W + 12) // 13)) < share
    on = np.kron(patch, np.ones((13, 13), bool))[:H, :W]
    return (np.where(on, stripes, 0.5) + 0.03 * rng.random((H, W))).astype(np.float32)


@pytest.mark.parametrize("H,W", [(33, 47), (96, 128), (113, 209), (304, 402)])
@pytest.mark.parametrize("shift", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("share", [1.0, 0.6, 0.05])
def test_textured_frames_match_oracle(oracle_lib, gpu, H, W, shift, share):
    import torch

    import imops_b200 as im
    m = _texture(H, W, share, seed=H + 3 * W + 7 * shift[0] + 11 * shift[1])
    ref = oracle_lib.amaze(m, "RGGB", shift=shift, clip_pt=1.0, precision="f32")
    out = im.demosaic_amaze(torch.from_numpy(m).to(gpu), "RGGB", shift=shift, clip_pt=1.0).cpu().numpy()
    assert np.array_equal(out, ref)
