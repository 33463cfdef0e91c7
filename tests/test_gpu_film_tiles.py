"""The reference film model at the sizes where its tiled kernels can go wrong:
frames smaller than a tile or a blur radius, sides one off a tile, and strips
wide enough for the real blur radii, over every emulsion layer count (1, 2,
3, 6, 7).  Against the CPU oracle within the film parity tolerance of
tests/test_gpu_film.py (1e-4 absolute in linear [0, 1]: f32 densities of up
to about 10 after the sum over layers, 1e-6 relative each, times ln 10)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-4
STOCKS = [0, 1, 3, 4, 5, 6]  # 1, 3, 6, 7, 3 (reversal) and 2 layers


def _scene(H, W, seed):
    rng = np.random.default_rng(seed)
    rel = rng.random((H, W, 3)) ** 2 * 1.2
    return (rel * (12.5 * 64.0)).astype(np.float32)


@pytest.mark.parametrize("stock", STOCKS)
@pytest.mark.parametrize("H,W", [(1, 1), (1, 70), (65, 1), (31, 65), (33, 129), (7, 6049), (70, 3001)])
def test_ragged_frames_match_oracle(oracle_lib, gpu, stock, H, W):
    import torch

    import imops_b200 as im
    x = _scene(H, W, seed=100 * stock + W)
    ref = oracle_lib.film_process(x, stock=stock, seed=11, output=1, grain=True, precision="f32")
    out = im.film_process(torch.from_numpy(x).to(gpu), stock=stock, seed=11, output=1, grain=True).cpu().numpy()
    assert np.isfinite(out).all()
    assert np.abs(out - ref).max() < TOL


@pytest.mark.parametrize("stock", STOCKS)
@pytest.mark.parametrize("H,W", [(1, 1), (33, 129), (9, 6049)])
def test_sub_stages_equal_the_whole_on_ragged_frames(gpu, stock, H, W):
    import torch

    import imops_b200 as im
    x = torch.from_numpy(_scene(H, W, seed=7 * stock + W)).to(gpu)
    ref = im.film_process(x.clone(), stock=stock, seed=5, output=1, grain=True)
    got = im.FilmStages(stock=stock, seed=5, output=1, grain=True).run(x.clone())
    assert torch.equal(got, ref)


@pytest.mark.parametrize("stock", [1, 2])
def test_develop_agrees_across_the_tile_radius_line(gpu, stock):
    """Flat planes develop to the same densities on both sides of the width
    above which the DIR blur no longer fits the tiles' halo (a flat plane's
    blur is the plane; f32 rounding of 33 taps and the exponential, 1e-5)."""
    import torch

    import imops_b200 as im
    st = im.FilmStages(stock=stock, grain=False)
    res = []
    for w in (11000, 13500):
        planes = torch.full((st.layers, 3, w), 0.37, device=gpu) * torch.arange(1, st.layers + 1, device=gpu)[:, None, None]
        dens, mask = st.develop(planes)
        assert float((dens - dens[:, :1, :1]).abs().max()) < 1e-5
        res.append(torch.cat([dens[:, 0, 0], mask[:, 0, 0]]))
    assert float((res[0] - res[1]).abs().max()) < 1e-5
