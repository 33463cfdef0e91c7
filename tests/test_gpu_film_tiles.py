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


def _noise_rows(seed, layer, y0, y1, W):
    """Unblurred grain of rows y0..y1-1: the sum of twelve SplitMix64 uniforms a pixel, minus 6."""
    m = (1 << 64) - 1
    golden = 0x9E3779B97F4A7C15
    y = np.arange(y0, y1, dtype=np.uint64)[:, None]
    x = np.arange(W, dtype=np.uint64)[None, :]
    base = np.uint64((seed * 0xD1B54A32D192ED03 + layer * golden) & m) + y + x * np.uint64((12 * golden) & m)
    acc = np.zeros(base.shape)
    for k in range(1, 13):
        z = base + np.uint64((k * golden) & m)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        acc += (z ^ (z >> np.uint64(31))).astype(np.float64) / 2.0 ** 64
    return acc - 6.0


@pytest.mark.parametrize("stock,H,W", [(2, 1500, 2100), (4, 1500, 2100), (1, 1500, 2100), (1, 300, 517), (6, 300, 517),
                                       (0, 216, 324), (1, 216, 324), (1, 480, 640), (6, 480, 640), (0, 800, 1200),
                                       (1, 800, 1200), (6, 864, 1296), (1, 864, 1296), (1, 683, 1024)])
def test_grain_fields_match_the_generator(gpu, stock, H, W):
    """The grain added to flat planes, against the generator in 64 bits, over
    rows that cross tile edges, for one block of six layers (2), six and one
    (4), three (1), two layers (6) and one (0), and every height of the tiles
    that smaller images take.  Up to
    the layer's amplitude the added densities are the blurred noise.  Error: two
    f32 roundings of an output below 0.5 (6e-8 each), and 1e-5 of the
    grain for the rounding of its blur and scale."""
    import torch

    import imops_b200 as im
    seed, y0, y1 = 12345, 20, 64
    st = im.FilmStages(stock=stock, seed=seed, grain=True)
    planes = torch.full((st.layers, H, W), 0.25, device=gpu)  # inside every layer's range
    out = st.grain(planes.clone()).cpu().numpy().astype(np.float64) - 0.25
    t = np.exp(-np.arange(-3, 4) ** 2 / 2.0)
    t /= t.sum()
    for e in range(st.layers):
        n = _noise_rows(seed, e, y0 - 3, y1 + 3, W)
        n = np.pad(n, ((0, 0), (3, 3)), mode="reflect")
        n = sum(t[k] * n[:, k:k + W] for k in range(7))
        n = sum(t[k] * n[k:k + y1 - y0] for k in range(7))
        got = out[e, y0:y1]
        scale = (got * n).sum() / (n * n).sum()
        assert scale > 0
        assert np.abs(got - scale * n).max() < 1e-5 * np.abs(got).max() + 1.2e-7
        assert abs(got.std() / out[e].std() - 1) < 0.05


@pytest.mark.parametrize("stock", STOCKS)
@pytest.mark.parametrize("output", [0, 1])
def test_capture_over_twelve_decades_matches_oracle(oracle_lib, gpu, stock, output):
    """Steps of exposure from below the capture LUT's first entry to above its
    last, so that every entry of every layer is read (and the ends clamp)."""
    import torch

    import imops_b200 as im
    steps = np.repeat(10.0 ** np.linspace(-7, 7, 141), 4)
    x = np.broadcast_to(steps[None, :, None], (9, steps.size, 3)).astype(np.float32).copy()
    ref = oracle_lib.film_process(x, stock=stock, seed=3, output=output, grain=False, precision="f32")
    out = im.film_process(torch.from_numpy(x).to(gpu), stock=stock, seed=3, output=output, grain=False).cpu().numpy()
    assert np.isfinite(out).all()
    assert np.abs(out - ref).max() < TOL


@pytest.mark.parametrize("H,W", [(1, 1), (5, 33), (31, 65), (33, 64), (97, 1200), (800, 1200), (1024, 1536), (1100, 1536)])
def test_preset_scan_matches_oracle_on_both_sides_of_its_block_rule(oracle_lib, gpu, H, W):
    """The 81-band preset with four rows a thread (few blocks) and sixteen."""
    import torch

    import imops_b200 as im
    x = (np.random.default_rng(H + W).random((H, W, 3)) ** 2).astype(np.float32)
    ref = oracle_lib.film_baseline(x, oracle_lib.baseline_params(grain_on=1, seed=9), precision="f64")
    out = im.film_process(torch.from_numpy(x).to(gpu), stock=im.STOCK_BASELINE81,
                          baseline=im.baseline_film_defaults(grain_on=1, seed=9)).cpu().numpy()
    assert np.abs(out - ref).max() < TOL


def test_positives_from_threads_and_streams(gpu):
    """A positive's mid-grey patch runs on a stream of the device's own, shared
    by all callers: frames of other sizes and stocks from four threads, each
    on its stream, give what each gives alone."""
    import threading

    import torch

    import imops_b200 as im
    work = [(1, 40, 61), (3, 300, 517), (6, 33, 129), (2, 64, 2050)]
    xs = [torch.from_numpy(_scene(h, w, seed=h)).to(gpu) for _, h, w in work]
    alone = [im.film_process(x.clone(), stock=st, seed=2, output=1, grain=True) for x, (st, _, _) in zip(xs, work)]
    torch.cuda.synchronize()
    bad = []

    def run(k):
        s = torch.cuda.Stream(gpu)
        with torch.cuda.stream(s):
            for _ in range(8):
                out = im.film_process(xs[k].clone(), stock=work[k][0], seed=2, output=1, grain=True)
                s.synchronize()
                if not torch.equal(out, alone[k]):
                    bad.append(k)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


@pytest.mark.parametrize("stock,H,W", [(1, 300, 680), (1, 300, 690), (0, 760, 808), (0, 760, 809), (2, 300, 343)])
def test_grain_beside_the_frame_matches_the_sub_stages(gpu, stock, H, W):
    """Negatives just below and above the size from which the grain fields run
    on the side stream, against the sub-stages, which never do; repeated, as
    each call's planes are the last one's."""
    import torch

    import imops_b200 as im
    x = torch.from_numpy(_scene(H, W, seed=stock + W)).to(gpu)
    ref = im.FilmStages(stock=stock, seed=5, output=0, grain=True).run(x.clone())
    for _ in range(4):
        assert torch.equal(im.film_process(x.clone(), stock=stock, seed=5, output=0, grain=True), ref)
