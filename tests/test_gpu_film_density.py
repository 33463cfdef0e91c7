"""Densities of thin exposures to a few units in the last place: below the
capture LUT's first entry (phi = 1e-4) a layer's developable fraction is that
entry, 2e-5 to 4e-4, and its density dmax f^(1/gamma), inhibited by the other
layers'.  On frames this narrow (millimetres a pixel) no blur has any reach.

Bound, relative: the power 2.1e-7 (the log2 of a mantissa good to 4e-8, times
1/gamma up to 2.94 and ln 2, 8e-8; the remainder's two roundings, 4e-8 and
1e-8; the exponential's, 8e-8), half a unit (6e-8) for the product with dmax,
the exponential of the inhibition and the product with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# per emulsion layer: mean grain size, its spread, capture k, gamma, dmax
LAYERS = {
    0: [(0.7, 0.35, 1.0, 0.65, 2.5)],
    1: [(0.55, 0.3, 4.2, 0.65, 2.2), (0.6, 0.32, 2.1, 0.65, 2.2), (0.7, 0.35, 1.35, 0.65, 2.2)],
    2: [(0.85, 0.35, 4.8, 0.54, 1.1), (0.42, 0.28, 2.2, 0.54, 1.1), (0.9, 0.35, 2.4, 0.54, 1.1),
        (0.45, 0.28, 1.1, 0.54, 1.1), (0.95, 0.35, 1.5, 0.54, 1.1), (0.48, 0.28, 0.7, 0.54, 1.1)],
    3: [(0.82, 0.32, 4.8, 0.58, 1.25), (0.38, 0.24, 6.5, 0.34, 1.9), (0.88, 0.32, 2.6, 0.58, 1.25),
        (0.4, 0.24, 3.6, 0.34, 1.9), (0.92, 0.32, 1.6, 0.58, 1.25), (0.42, 0.24, 2.4, 0.34, 1.9)],
    4: [(0.82, 0.33, 4.5, 0.56, 1.1), (0.4, 0.28, 2.1, 0.56, 1.1), (0.5, 0.3, 2.0, 0.56, 0.5),
        (0.88, 0.34, 2.3, 0.56, 1.1), (0.44, 0.28, 1.1, 0.56, 1.1), (0.92, 0.34, 1.4, 0.56, 1.1),
        (0.46, 0.28, 0.7, 0.56, 1.1)],
    6: [(0.95, 0.38, 2.2, 0.70, 1.5), (0.45, 0.28, 0.9, 0.70, 1.5)],
}
# inhibition: row i, column j is how much layer i's density inhibits layer j
DIR = {
    0: [[0.0]],
    1: [[0.02, 0.05, 0.03],
        [0.05, 0.02, 0.06],
        [0.03, 0.06, 0.02]],
    2: [[0.02, 0.01, 0.04, 0.02, 0.03, 0.01],
        [0.01, 0.01, 0.02, 0.01, 0.02, 0.01],
        [0.04, 0.02, 0.02, 0.01, 0.05, 0.02],
        [0.02, 0.01, 0.01, 0.01, 0.02, 0.01],
        [0.03, 0.01, 0.05, 0.02, 0.02, 0.01],
        [0.01, 0.01, 0.02, 0.01, 0.01, 0.01]],
    3: [[0.03, 0.02, 0.09, 0.04, 0.07, 0.03],
        [0.02, 0.02, 0.04, 0.02, 0.04, 0.02],
        [0.09, 0.04, 0.03, 0.02, 0.1, 0.04],
        [0.04, 0.02, 0.02, 0.02, 0.04, 0.02],
        [0.07, 0.03, 0.1, 0.04, 0.03, 0.02],
        [0.03, 0.02, 0.04, 0.02, 0.02, 0.02]],
    4: [[0.02, 0.01, 0.03, 0.04, 0.02, 0.03, 0.01],
        [0.01, 0.01, 0.02, 0.02, 0.01, 0.02, 0.01],
        [0.03, 0.02, 0.02, 0.06, 0.03, 0.04, 0.02],
        [0.04, 0.02, 0.05, 0.02, 0.01, 0.05, 0.02],
        [0.02, 0.01, 0.02, 0.01, 0.01, 0.02, 0.01],
        [0.03, 0.01, 0.04, 0.05, 0.02, 0.02, 0.01],
        [0.01, 0.01, 0.02, 0.02, 0.01, 0.01, 0.01]],
    6: [[0.03, 0.02],
        [0.02, 0.02]],
}


@pytest.mark.parametrize("stock", sorted(LAYERS))
def test_thin_densities(oracle_lib, gpu, stock):
    import torch

    import imops_b200 as im
    st = im.FilmStages(stock=stock, grain=False, shutter=0.01)
    dens, _ = st.develop(torch.full((st.layers, 4, 6), 1e-6, device=gpu))
    got = dens.cpu().numpy().astype(np.float64)
    want = []
    for mean, sigma, k, gamma, dmax in LAYERS[stock]:
        f = np.float32(oracle_lib.lut_build_sample(np.log(mean), sigma, k, 1e-6))  # the LUT's first entry
        want.append(np.float64(np.float32(dmax)) * np.float64(f) ** np.float64(np.float32(1.0) / np.float32(gamma)))
    want = np.array(want)
    want = want * np.exp(-want @ np.array(DIR[stock]))
    rel = np.abs(got / want[:, None, None] - 1)
    assert rel.max() <= 2.1e-7 + 3 * 6e-8, rel.max(axis=(1, 2))
