"""The reference film model at real blur radii on frames of more than one row of
tiles, with structure: inner tiles (copied 16 bytes a lane) and edge tiles of
every template radius, and the launches of their own that take over where a
blur outgrows the tiles, against results in 64 bits."""
import numpy as np
import pytest

from test_gpu_film_density import DIR, LAYERS

pytestmark = pytest.mark.gpu

# A pixel's transmittance T = 10^-D moves by T ln(10) dD, and T D ln(10) is at
# most 1/e a channel: relative errors of 1e-6 in the densities (f32 sums of up
# to 2 x 33 taps, the LUT's place and the power, 2e-7 each or less; 2 to 7
# layers) stay below 2e-6.  The inversion divides by T: its relative error,
# ln(10) D 1e-6 at densities of 2, times outputs of up to 1.5, below 1e-5.
NEGATIVE, POSITIVE = 2e-6, 1e-5

FRAMES = [(0, 6048), (1, 6048), (2, 6048), (3, 6048), (4, 6048), (5, 6048), (6, 6048),
          (1, 9596),    # inhibition radius 12
          (2, 10968),   # 15
          (4, 11812),   # 14
          (6, 15356),   # 16, adjacency 8
          (5, 19196),   # 13, grain blur 5
          (3, 13716),   # 17: the inhibition's blurs are launches of their own
          (0, 19204),   # adjacency 9: a launch of its own
          (0, 48004),   # local scatter 9 too
          (0, 63996)]   # the widest grain blur, 16


@pytest.mark.parametrize("stock,W", FRAMES)
def test_wide_frames_match_64_bits(oracle_lib, gpu, stock, W):
    import torch

    import imops_b200 as im
    H = 84 if W < 20000 else 40
    x = (np.random.default_rng(stock + W).random((H, W, 3)) ** 2 * 960).astype(np.float32)
    for output, bar in ((0, NEGATIVE), (1, POSITIVE)):
        ref = oracle_lib.film_process(x, stock=stock, seed=11, output=output, grain=output == 0, precision="f64")
        out = im.film_process(torch.from_numpy(x).to(gpu), stock=stock, seed=11, output=output,
                              grain=output == 0).cpu().numpy()
        assert np.isfinite(out).all()
        assert np.abs(out - ref).max() < bar


def _taps(sigma):
    sigma = np.float64(np.float32(sigma))
    r = max(int(np.ceil(3 * sigma)), 1)
    t = np.exp(-np.arange(-r, r + 1) ** 2 / (2 * sigma * sigma))
    return r, t / t.sum()


def _blur(v, sigma):
    r, t = _taps(sigma)
    H, W = v.shape
    p = np.pad(v, ((0, 0), (r, r)), mode="reflect")
    p = sum(t[k] * p[:, k:k + W] for k in range(2 * r + 1))
    p = np.pad(p, ((r, r), (0, 0)), mode="reflect")
    return sum(t[k] * p[k:k + H] for k in range(2 * r + 1))


# inhibition and adjacency blurs in micrometres, adjacency strength
DIFFUSION = {2: (16.0, 7.0, 0.3), 4: (14.0, 6.5, 0.32)}


@pytest.mark.parametrize("stock", sorted(DIFFUSION))
@pytest.mark.parametrize("radius", range(1, 19))
def test_development_at_every_radius(oracle_lib, gpu, stock, radius):
    """Densities up to 1.1 (and the masks), each good to about 1e-6: 3e-6."""
    import torch

    import imops_b200 as im
    dir_um, adj_um, beta = DIFFUSION[stock]
    H, W = 84, int((radius - 0.25) * 36000 / (3 * dir_um)) // 4 * 4
    pitch = 36000.0 / W
    assert _taps(dir_um / pitch)[0] == radius
    st = im.FilmStages(stock=stock, grain=False, shutter=0.01)
    rng = np.random.default_rng(radius)
    x = (10.0 ** rng.uniform(-2, 2.5, (st.layers, H, W))).astype(np.float32)
    dens, mask = st.develop(torch.from_numpy(x).to(gpu))
    knots = np.linspace(-4.0, 8.0, 64)
    D0, want_mask = [], []
    for e, (_, _, _, gamma, dmax) in enumerate(LAYERS[stock]):
        lut = [oracle_lib.lut_sample(stock, e, 10.0 ** v) for v in knots]
        q = np.interp(np.log10(x[e].astype(np.float64)), knots, lut) ** (1.0 / np.float64(np.float32(gamma)))
        D0.append(np.float64(np.float32(dmax)) * q)
        want_mask.append(0.4 * dmax * (1.0 - q))
    blurred = [_blur(d, dir_um / pitch) for d in D0]
    m = np.array(DIR[stock])
    for j, d in enumerate(D0):
        d = d * np.exp(-sum(m[i, j] * b for i, b in enumerate(blurred)))
        d = d + beta * (d - _blur(d, adj_um / pitch))
        assert np.abs(dens[j].cpu().numpy() - d).max() < 3e-6
        assert np.abs(mask[j].cpu().numpy() - want_mask[j]).max() < 3e-6
