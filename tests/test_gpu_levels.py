"""Black/white scaling of every u16 value, bit for bit the f32 division, for
level pairs on both sides of the rule that replaces the division (one usable
pair for all cells) -- through imops_scale_u16 and through the X-Trans / Bayer
develop, which scales while it stages, at odd crops and frame edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAIRS = [(600.0, 16383.0), (0.0, 65535.0), (0.0, 1.0), (511.75, 4095.0), (2047.3, 16000.6), (64.0, 1023.0),
         (0.001, 3.7), (-12.5, 255.0), (1e-12, 100.0), (100.0, 50.0), (0.0, 3e7)]


def _ref(v, b, w):
    return (v.astype(np.float32) - np.float32(b)) / (np.float32(w) - np.float32(b))


@pytest.mark.parametrize("black,white", PAIRS)
def test_scale_every_value(gpu, black, white):
    import torch

    import imops_b200 as im
    v = np.arange(65536, dtype=np.uint16).reshape(256, 256)
    raw = torch.from_numpy(v.view(np.int16)).to(gpu)
    got = im.scale_u16(raw, (0, 0, 256, 256), black, white).cpu().numpy()
    assert np.array_equal(got, _ref(v, black, white))
    got = im.scale_u16(raw, (3, 5, 250, 247), black, white).cpu().numpy()
    assert np.array_equal(got, _ref(v[5:252, 3:253], black, white))


CELLS = {"RGGB": 2, "GGRGGBGGBGGRBRGRBGGGBGGRGGRGGBRBGBRG": 6}


@pytest.mark.parametrize("pattern", sorted(CELLS))
@pytest.mark.parametrize("black,white", PAIRS[:6] + [(None, None)])
@pytest.mark.parametrize("crop", [(0, 0, 300, 131), (7, 3, 193, 8), (1, 2, 5, 9), (4, 1, 400, 1)])
def test_develop_equals_scaling_then_mean(gpu, pattern, black, white, crop):
    import torch

    import imops_b200 as im
    p = CELLS[pattern]
    rng = np.random.default_rng(3)
    raw = torch.from_numpy(rng.integers(0, 65536, (140, 410), dtype=np.uint16).view(np.int16)).to(gpu)
    if black is None:  # levels of their own for every cell
        black = rng.uniform(0, 900, p * p).tolist()
        white = rng.uniform(12000, 16383, p * p).tolist()
    x, y, w, h = crop
    params = im.DevelopParams()
    params.demosaic, params.cfa, params.clip_pt, params.n_gain = im.DEMOSAIC_MARKESTEIJN, pattern.encode(), 1.0, 1
    params.ev[0], params.target, params.film = 0.3, im.CS_ACESCG, 0
    wb, calib = [2.0, 1.0, 1.5, 0.0], [0.7, -0.1, -0.1, -0.4, 1.2, 0.2, -0.1, 0.2, 0.6]
    for i in range(4):
        params.wb[i] = wb[i]
    for i in range(9):
        params.calib_d65[i] = calib[i]
    got = im.develop_u16(raw, crop, black, white, params, period=(p, p))
    m = im.scale_u16(raw, crop, black, white, period=(p, p))
    ref = im.demosaic_markesteijn(m, pattern, shift=(x, y))
    im.cfa_coeffs(ref, wb)
    im.exp(ref, 0.3)
    im.camera_cst(ref, calib, im.CS_ACESCG)
    assert torch.equal(got, ref)
