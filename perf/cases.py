"""The work this framework is used for, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program has in hand before the call
(seeded inputs on the GPU, parameters, a parsed pipeline), `run` is one pass through the public
entry points, `work` the bytes and operations that the result cannot do without, and `exact` the
same result in 64 bits from plain torch, for the kinds whose result is a smooth function of the
input.  AMaZE and the 3-pass X-Trans demosaic have no such value: both are defined by f32
comparisons (which estimate is kept, which direction wins), and a comparison that falls the other
way in 64 bits gives another, equally valid pixel.

Kinds
  develop   a u16 sensor frame to ACEScg, optionally through the 81-bin film preset: the import
            of a raw file (Bayer: AMaZE; X-Trans: the 3x3 same-colour mean)
  xtrans3   the 3-pass directional X-Trans demosaic: the high-quality export of an X-Trans frame
  film      a film simulation on a developed image, as an editor does when a stock or a seed
            changes (the developed image is kept, so the pass works on a copy)
  fit       one gradient step of the 24-parameter colour + film model over a batch of frames
  display   the display stages after the scan (tone map, grading, output encoding)
  preview   the interactive path: a quad-sampled frame, colour, film and output encoding
  pipeline  the embedding interface: host buffers in and out, images on the device between modules
"""
from __future__ import annotations

import math

import numpy as np
import torch

import imops_b200 as im
from imops_b200 import synthetic
from imops_b200.pipeline import Image, make_meta, parse_config, run_pixel_pipeline

DEV = "cuda"
BLACK, WHITE = synthetic.BLACK, synthetic.WHITE
WB = synthetic.WB
CALIB = synthetic.CALIB_D65
BAYER, XTRANS = "RGGB", synthetic.XTRANS
SUNNY16 = 12.5 * 64.0  # relative to absolute luminance where shutter * ISO = 1 and N = 8


def listed():
    return [
        # the import of a 24 MP Bayer raw file through the film preset (the benchmark's frame size)
        dict(name="bayer_24mp_film", kind="develop", sensor="bayer", w=6048, h=4024, x=0, y=0, film=True, grain=True),
        # a crop at an odd origin, developed to ACEScg only: a ragged Bayer frame of a few megapixels
        dict(name="bayer_3mp_crop", kind="develop", sensor="bayer", w=2141, h=1423, x=13, y=7, film=False, grain=False),
        # the import of a 24 MP X-Trans raw file
        dict(name="xtrans_24mp", kind="develop", sensor="xtrans", w=6032, h=4032, x=4, y=2, film=False, grain=False),
        # the high-quality demosaic of the same frame
        dict(name="xtrans3_24mp", kind="xtrans3", w=6032, h=4032, sx=0, sy=0),
        # the 81-bin preset re-run on a 12.6 MP image
        dict(name="film81_12mp", kind="film", stock="baseline81", w=4096, h=3072, grain=True, positive=False),
        # a reference stock at full size: six emulsion layers, every spatial effect, grain
        dict(name="portra_24mp", kind="film", stock="portra400", w=6048, h=4024, grain=True, positive=False),
        # a three-layer stock inverted to a positive on a ragged 8 MP image
        dict(name="colorneg_8mp", kind="film", stock="colorneg200", w=3465, h=2311, grain=True, positive=True),
        # a parameter fit: eight 2048x1365 frames a step
        dict(name="fit_8x2048", kind="fit", w=2048, h=1365, images=8, render=False),
        # forward and adjoint of one full frame
        dict(name="fit_24mp", kind="fit", w=6048, h=4024, images=1, render=True),
        # the display stages of a full frame
        dict(name="display_24mp", kind="display", w=6048, h=4024, look="filmic"),
        # the smallest calls: a quarter-size preview, where launches and latency count
        dict(name="preview_1mp", kind="preview", w=5184, h=3456, factor=4),
        # the embedding interface from host buffers, upload and download included
        dict(name="pipeline_6mp", kind="pipeline", w=3008, h=2008),
    ]


def _size(rng, lo_mp, hi_mp, least=160):
    """Width and height of lo..hi megapixels (log-uniform) at an aspect of 1:1 to 2:1, any parity."""
    mp = math.exp(rng.uniform(math.log(lo_mp), math.log(hi_mp))) * 1e6
    aspect = rng.uniform(1.0, 2.0)
    w = max(least, int(math.sqrt(mp * aspect)))
    h = max(least, int(math.sqrt(mp / aspect)))
    return w, h


def _amaze_size(v):
    """AMaZE refuses sides of 1..15 modulo 96 (the reference's tile fill runs past its buffer there)."""
    return v + 16 - v % 96 if 1 <= v % 96 <= 15 else v


def draw(rng):
    kind = rng.choice(["develop", "develop", "xtrans3", "film", "film", "fit", "display", "preview", "pipeline"])
    if kind == "develop":
        sensor = rng.choice(["bayer", "xtrans"])
        w, h = _size(rng, 0.3, 23.0)
        if sensor == "bayer":
            w, h = _amaze_size(w), _amaze_size(h)
        film = rng.random() < 0.5
        return dict(kind=kind, sensor=sensor, w=w, h=h, x=rng.randrange(24), y=rng.randrange(24), film=film,
                    grain=film and rng.random() < 0.7)
    if kind == "xtrans3":
        w, h = _size(rng, 0.3, 23.0)
        return dict(kind=kind, w=w, h=h, sx=rng.randrange(6), sy=rng.randrange(6))
    if kind == "film":
        w, h = _size(rng, 0.3, 23.0)
        return dict(kind=kind, stock=rng.choice(sorted(STOCK_IDS)), w=w, h=h, grain=rng.random() < 0.7,
                    positive=rng.random() < 0.5)
    if kind == "fit":
        images = rng.randrange(1, 5)
        w, h = _size(rng, 0.3, 22.0 / images)
        return dict(kind=kind, w=w, h=h, images=images, render=rng.random() < 0.5)
    if kind == "display":
        w, h = _size(rng, 0.3, 23.0)
        return dict(kind=kind, w=w, h=h, look=rng.choice(["filmic", "grade"]))
    if kind == "preview":
        w, h = _size(rng, 6.0, 23.0)
        return dict(kind=kind, w=w, h=h, factor=rng.choice([2, 4, 8]))
    w, h = _size(rng, 0.3, 5.9)
    return dict(kind=kind, w=_amaze_size(w), h=_amaze_size(h))


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _scene(h, w, seed):
    """Scene-linear RGB: smooth gradients, sinusoidal texture of 2 to 40 px, and a few bright lights
    whose cores exceed diffuse white (1.0), as a photograph has them."""
    rng = np.random.default_rng(seed)
    y = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    x = torch.arange(w, device=DEV, dtype=torch.float32)[None, :]
    waves = torch.zeros((h, w), device=DEV)
    for _ in range(6):
        period, th, ph = rng.uniform(2.0, 40.0), rng.uniform(0, np.pi), rng.uniform(0, 2 * np.pi)
        k = 2 * np.pi / period
        waves += rng.uniform(0.02, 0.08) * torch.sin((x * math.cos(th) + y * math.sin(th)) * k + ph)
    lights = torch.zeros((h, w), device=DEV)
    for _ in range(12):
        r = rng.uniform(0.004, 0.03) * min(h, w) + 1.0
        d2 = (x - rng.uniform(0, w)) ** 2 + (y - rng.uniform(0, h)) ** 2
        lights += rng.uniform(0.5, 4.0) * torch.exp(-d2 / (2 * r * r))
    out = torch.empty((h, w, 3), device=DEV)
    for c in range(3):
        a, bx, by = rng.uniform(0.10, 0.35), rng.uniform(-0.2, 0.25), rng.uniform(-0.2, 0.25)
        out[..., c] = a + (bx / w) * x + (by / h) * y + waves * rng.uniform(0.6, 1.0) + lights * rng.uniform(0.7, 1.0)
    return out.clamp_(min=0.0)


def _raw(h, w, seed, pattern, period):
    """A 14-bit sensor frame of the scene: channels divided by their white balance, shot and read
    noise, saturation at the white level."""
    sc = _scene(h, w, seed)
    codes = torch.tensor(["RGB".index(c) for c in pattern], device=DEV).reshape(period, period)
    col = codes.repeat(-(-h // period), -(-w // period))[:h, :w]
    sig = torch.gather(sc, 2, col[..., None])[..., 0]
    gain = torch.tensor([1.0 / WB[0], 1.0 / WB[1], 1.0 / WB[2]], device=DEV)
    sig = sig * gain[col] * (WHITE - BLACK)
    noise = torch.randn((h, w), generator=_gen(seed), device=DEV)
    v = sig + noise * torch.sqrt(2.0 * sig + 9.0) + BLACK
    return v.round_().clamp_(0, WHITE).to(torch.int32).to(torch.uint16)


def _mosaic(h, w, seed, pattern, period):
    return (_raw(h, w, seed, pattern, period).to(torch.float32) - BLACK) / (WHITE - BLACK)


def _image(h, w, seed):
    """A developed image: the scene with a little sensor noise (slightly negative in the shadows)."""
    rgb = _scene(h, w, seed)
    return rgb.add_(torch.randn((h, w, 3), generator=_gen(seed), device=DEV), alpha=0.004)


def _theta(seed):
    return torch.tensor(synthetic.film_grad_perturbed(seed), dtype=torch.float64, device=DEV)


STOCK_IDS = {"baseline81": im.STOCK_BASELINE81, "colorneg200": im.STOCK_COLORNEG200,
             "portra400": im.STOCK_PORTRA400, "trix400": im.STOCK_TRIX400}

PIPELINE = """
[[pipeline_modules]]
name = "Demosaic"
algorithm = "amaze"
[[pipeline_modules]]
name = "CFACoeffs"
[[pipeline_modules]]
name = "CST"
target_color_space = "AcesCg"
[[pipeline_modules]]
name = "Film"
stock = "Baseline81"
film_format = "Film35mm"
seed = 1002
output = "NegativeLinear"
"""


def _film_seed(seed):
    return 1 + seed % 100003


def _fit_inputs(case, seed):
    """Camera RGB of each frame and the target it is fitted to: the frame through the model with
    perturbed parameters, in plain torch."""
    truth = _theta(7)
    xs, ts = [], []
    for i in range(case["images"]):
        x = _scene(case["h"], case["w"], seed + i)
        x = (x / torch.tensor(WB[:3], device=DEV)).clamp_(max=1.0).contiguous()
        xs.append(x)
        ts.append(_model(x, truth.float(), torch.float32))
    return xs, ts


def prepare(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    s = {"case": case}
    if kind == "develop":
        pattern, period = (BAYER, 2) if case["sensor"] == "bayer" else (XTRANS, 6)
        s["raw"] = _raw(h + case["y"] + 5, w + case["x"] + 11, seed, pattern, period)
        p = im.DevelopParams()
        p.demosaic = im.DEMOSAIC_AMAZE if case["sensor"] == "bayer" else im.DEMOSAIC_MARKESTEIJN
        p.cfa, p.clip_pt, p.n_gain, p.target, p.film = pattern.encode(), 1.0, 0, im.CS_ACESCG, int(case["film"])
        for i in range(4):
            p.wb[i] = WB[i]
        for i in range(9):
            p.calib_d65[i] = CALIB[i]
        p.film_params = im.FilmParams(im.STOCK_BASELINE81, 0, 1, 0, -1.0, int(case["grain"]))
        p.baseline = im.baseline_film_defaults(seed=_film_seed(seed), grain_on=int(case["grain"]))
        s["params"] = p
    elif kind == "xtrans3":
        s["mosaic"] = _mosaic(h, w, seed, XTRANS, 6)
    elif kind == "film":
        x = _image(h, w, seed)
        s["rgb"] = x if case["stock"] == "baseline81" else x.mul_(SUNNY16)
        s["seed"] = _film_seed(seed)
    elif kind == "fit":
        s["x"], s["target"] = _fit_inputs(case, seed)
        s["theta"] = im.FilmGradParams.from_vector(synthetic.film_grad_base())
        s["grad"] = torch.zeros(25, dtype=torch.float64, device=DEV)
        s["scale"] = 1.0 / (3 * case["images"] * w * h)
    elif kind == "display":
        s["rgb"] = _image(h, w, seed)
    elif kind == "preview":
        s["mosaic"] = _mosaic(h, w, seed, BAYER, 2)
        s["baseline"] = im.baseline_film_defaults(seed=_film_seed(seed))
    elif kind == "pipeline":
        s["raw"] = _raw(h, w, seed, BAYER, 2).cpu().numpy()
        s["meta"] = make_meta(cfa=BAYER, wb=WB, calibration=CALIB, black=BLACK, white=WHITE)
        s["pipeline"] = parse_config(PIPELINE)
    return s


# ---- one pass -----------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "develop":
        return im.develop_u16(s["raw"], (case["x"], case["y"], case["w"], case["h"]), BLACK, WHITE, s["params"])
    if kind == "xtrans3":
        return im.demosaic_markesteijn3(s["mosaic"], XTRANS, shift=(case["sx"], case["sy"]))
    if kind == "film":
        img = s["rgb"].clone()
        if case["stock"] == "baseline81":
            return im.film_process(img, stock=im.STOCK_BASELINE81,
                                   baseline=im.baseline_film_defaults(seed=s["seed"], grain_on=int(case["grain"])))
        output = im.FILM_POSITIVE_LINEAR if case["positive"] else im.FILM_NEGATIVE_LINEAR
        return im.film_process(img, stock=STOCK_IDS[case["stock"]], seed=s["seed"], output=output, grain=case["grain"])
    if kind == "fit":
        # an optimiser with f32 parameters takes the step's gradient and loss in f32
        out = {}
        if case["render"]:
            out["render"] = im.param_forward(s["x"][0], s["theta"])
        s["grad"].zero_()
        for x, t in zip(s["x"], s["target"]):
            im.param_backward(x, s["theta"], s["grad"], target=t, loss_scale=s["scale"])
        g = s["grad"].to(torch.float32)
        out["grad"], out["loss"] = g[:24], g[24:]
        return out
    if kind == "display":
        img = s["rgb"].clone()
        if case["look"] == "filmic":
            im.exp(img, 0.5)
            im.sigmoid_tone_map(img)
            im.cst(img, im.CS_ACESCG, im.CS_LINEAR_SRGB)
            return im.gamma(img, 2.2)
        im.contrast(img.clamp_(min=0.0), 1.2)
        im.lch(img, im.CS_ACESCG, 1.02, 1.15, 1.0)
        return im.cst(img, im.CS_ACESCG, im.CS_SRGB)
    if kind == "preview":
        img = im.demosaic_quad(s["mosaic"], BAYER, case["factor"])
        im.cfa_coeffs(img, WB)
        im.camera_cst(img, CALIB, im.CS_ACESCG)
        im.film_process(img, stock=im.STOCK_BASELINE81, baseline=s["baseline"])
        return im.cst(img, im.CS_ACESCG, im.CS_SRGB)
    img = Image.from_u16(s["raw"], s["meta"])
    return run_pixel_pipeline(img, s["pipeline"]).rgb_f32()


def work(case):
    """Bytes: each input read once, each output written once.  Operations: the arithmetic of the
    method per pixel (a transcendental counted as one)."""
    kind, n = case["kind"], case["w"] * case["h"]
    mean, colour, amaze, xt3 = 14, 36, 450, 1400
    film81 = 2 * 129 * 2 + 81 * 13 + 60  # separable halation, scan, exposures and curves
    grain = 12 * 10 + 3 * 2 * 14         # draws shared by the layers, blur
    if kind == "develop":
        f = (amaze if case["sensor"] == "bayer" else mean) + colour
        f += (film81 + (grain if case["grain"] else 0)) if case["film"] else 0
        return {"bytes": 14 * n, "flops": f * n}
    if kind == "xtrans3":
        return {"bytes": 16 * n, "flops": xt3 * n}
    if kind == "film":
        if case["stock"] == "baseline81":
            return {"bytes": 24 * n, "flops": (film81 + (grain if case["grain"] else 0)) * n}
        st = _reference_stock(case["stock"], case["w"])
        E = st["E"]
        taps = sum(2 * 2 * (2 * _radius(v) + 1) * c for v, c in
                   ((st["s_local"], E), (st["s_wide"], 1), (st["s_dir"], E), (st["s_adj"], E)))
        f = taps + E * (6 + 20 + 2 * E) + 16 * (4 * E + 7) + (E * (120 + 28) if case["grain"] else 0)
        return {"bytes": 24 * n, "flops": f * n}
    if kind == "fit":
        back = 3 * 2 * 129 * 2 + 81 * 32 + 150
        b = case["images"] * 24 * n + (24 * n if case["render"] else 0)
        return {"bytes": b, "flops": (case["images"] * back + (film81 if case["render"] else 0)) * n}
    if kind == "display":
        return {"bytes": 24 * n, "flops": (200 if case["look"] == "filmic" else 150) * n}
    if kind == "preview":
        m = (case["w"] // case["factor"]) * (case["h"] // case["factor"])
        return {"bytes": (16 + 12) * m, "flops": (film81 + grain + 100) * m}
    return {"bytes": 14 * n, "flops": (amaze + colour + film81 + grain) * n}


# ---- the same results in 64 bits, plain torch ------------------------------------------------------

XYZ2AP1 = np.array([[1.6410233797, -0.3248032942, -0.2364246952], [-0.6636628587, 1.6153315917, 0.0167563477],
                    [0.0117218943, -0.0082844165, 0.9883948585]])
AP12XYZ = np.array([[0.6624541811, 0.1340042065, 0.1561876870], [0.2722287168, 0.6740817658, 0.0536895174],
                    [-0.0055746495, 0.0040607335, 1.0103391003]])
XYZ2LIN = np.array([[12831 / 3959, -329 / 214, -1974 / 3959], [-851781 / 878810, 1648619 / 878810, 36519 / 878810],
                    [705 / 12673, -2585 / 12673, 705 / 667]])
LIN2XYZ = np.array([[506752 / 1228815, 87881 / 245763, 12673 / 70218],
                    [87098 / 409605, 175762 / 245763, 12673 / 175545],
                    [7918 / 409605, 87881 / 737289, 1001167 / 1053270]])
LUMA = AP12XYZ[1]
OK_M1 = np.array([[0.4122214708, 0.5363325363, 0.0514459929], [0.2119034982, 0.6806995451, 0.1073969566],
                  [0.0883024619, 0.2817188376, 0.6299787005]])
OK_M2 = np.array([[0.2104542553, 0.7936177850, -0.0040720468], [1.9779984951, -2.4285922050, 0.4505937099],
                  [0.0259040371, 0.7827717662, -0.8086757660]])
OK_M2I = np.array([[1.0, 0.3963377774, 0.2158037573], [1.0, -0.1055613458, -0.0638541728],
                   [1.0, -0.0894841775, -1.2914855480]])
OK_M1I = np.array([[4.0767416621, -3.3077115913, 0.2309699292], [-1.2684380046, 2.6097574011, -0.3413193965],
                   [-0.0041960863, -0.7034186147, 1.7076147010]])


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=DEV)


def _mat(v, m):
    """Matrix m (3x3) applied to the last axis."""
    return v @ _t(m).T


def _f32(a):
    """Values as the C interface holds them."""
    return np.asarray(a, np.float32).astype(np.float64)


def _camera_matrix():
    """Camera RGB to XYZ: the pseudo-inverse of the calibration scaled to map D65 white to 1."""
    c = _f32(CALIB).reshape(3, 3)
    white = c @ np.array([0.95042, 1.0, 1.08890])
    return np.linalg.pinv(c / white[:, None])


def _reflect(i, n):
    """Mirror without repeating the edge sample, as often as it takes."""
    if n == 1:
        return np.zeros_like(i)
    i = np.abs(i) % (2 * n - 2)
    return np.where(i >= n, 2 * n - 2 - i, i)


def _blur_axis(p, taps, dim):
    r, n = (len(taps) - 1) // 2, p.shape[dim]
    idx = torch.as_tensor(_reflect(np.arange(-r, n + r), n), device=p.device)
    pad = p.index_select(dim, idx)
    if isinstance(taps, torch.Tensor):  # differentiable in the taps
        out = 0.0
        for k in range(2 * r + 1):
            out = out + taps[k] * pad.narrow(dim, k, n)
        return out
    out = torch.zeros_like(p)
    for k in range(2 * r + 1):
        out.add_(pad.narrow(dim, k, n), alpha=float(taps[k]))
    return out


def _blur(p, taps):
    return _blur_axis(_blur_axis(p, taps, 1), taps, 0)


def _radius(sigma):
    return max(math.ceil(3.0 * sigma), 1) if sigma >= 1e-3 else 0


def _gauss(sigma, r=None):
    r = _radius(np.float32(sigma)) if r is None else r
    x = np.arange(-r, r + 1, dtype=np.float64)
    g = np.exp(-x * x / (2.0 * sigma * sigma))
    return g / g.sum()


def _srl(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >= 1 << 63 else v


def _grain(h, w, seed, layer, taps):
    """The blurred grain field of one layer and 1 / its RMS: twelve uniforms a pixel from the
    SplitMix64 stream of (seed, layer, row)."""
    golden = 0x9E3779B97F4A7C15
    out = torch.empty((h, w), dtype=torch.float64, device=DEV)
    x = torch.arange(w, device=DEV, dtype=torch.int64)[None, :] * _i64(12 * golden)
    rows = max(1, (1 << 22) // w)
    for y0 in range(0, h, rows):
        y = torch.arange(y0, min(h, y0 + rows), device=DEV, dtype=torch.int64)[:, None]
        z0 = x + y + _i64(seed * 0xD1B54A32D192ED03 + layer * golden)
        acc = 0.0
        for k in range(1, 13):
            z = z0 + _i64(k * golden)
            z = (z ^ _srl(z, 30)) * _i64(0xBF58476D1CE4E5B9)
            z = (z ^ _srl(z, 27)) * _i64(0x94D049BB133111EB)
            z = z ^ _srl(z, 31)
            acc = acc + _srl(z, 32).double() * 2.0 ** -32 + (z & 0xFFFFFFFF).double() * 2.0 ** -64
        out[y0:y0 + rows] = acc - 6.0
    out = _blur(out, taps)
    var = float((out * out).mean())
    return out, (1.0 / math.sqrt(var) if var > 1e-12 else 1.0)


# The 81-bin preset: 380..780 nm in steps of 5, three Gaussian layers.
_TABLES = {}


def _preset():
    if _TABLES:
        return _TABLES
    lam = 380.0 + 5.0 * np.arange(81)
    trap = np.full(81, 5.0)
    trap[0] = trap[-1] = 2.5

    def lobe(mu, s1, s2):
        t = (lam - mu) / np.where(lam < mu, s1, s2)
        return np.exp(-0.5 * t * t)

    cmf = np.stack([1.056 * lobe(599.8, 37.9, 31.0) + 0.362 * lobe(442.0, 16.0, 26.7) - 0.065 * lobe(501.1, 20.4, 26.2),
                    0.821 * lobe(568.8, 46.9, 40.5) + 0.286 * lobe(530.9, 16.3, 31.1),
                    1.217 * lobe(437.0, 11.8, 36.0) + 0.681 * lobe(459.0, 26.0, 13.8)])
    peak = np.array([450.0, 550.0, 650.0])[:, None]
    basis = np.exp(-0.5 * ((lam - peak) / 40.0) ** 2)
    sens = np.exp(-0.5 * ((lam - peak) / np.array([35.0, 40.0, 45.0])[:, None]) ** 2)
    minv = np.linalg.inv(XYZ2AP1 @ (cmf * trap) @ basis.T)
    w1 = np.maximum(0.0, minv.sum(1))
    A = (basis * trap) @ sens.T / (((w1 @ basis) * trap) @ sens.T)
    white = XYZ2AP1 @ (cmf * trap).sum(1)
    eps = np.exp(-0.5 * ((lam - peak) / np.array([40.0, 40.0, 45.0])[:, None]) ** 2)
    _TABLES.update(minv=minv, A=A, eps=eps * math.log2(10.0), C=((XYZ2AP1 @ cmf) * trap / white.max()).T,
                   bleed=_f32([0.20, 0.45, 1.0]), dmax=_f32([2.0, 2.1, 2.2]), k=_f32([2.3, 2.5, 2.7]),
                   x0=_f32([-0.70, -0.73, -0.76]), strength=_f32(0.15), threshold=_f32(0.8), grain=_f32(0.02))
    return _TABLES


def _scan(D, eps, C, rows=1 << 20):
    """sum over the bins of C 2^(-D . eps), in chunks of pixels."""
    flat = D.reshape(-1, D.shape[-1])
    out = torch.empty((flat.shape[0], 3), dtype=D.dtype, device=D.device)
    for i in range(0, flat.shape[0], rows):
        out[i:i + rows] = torch.exp2(-(flat[i:i + rows] @ eps)) @ C
    return out.reshape(*D.shape[:-1], 3)


def _film81(rgb, seed, grain):
    T = _preset()
    h, w = rgb.shape[:2]
    e = _mat(rgb, T["minv"]).clamp_(min=0.0) @ _t(T["A"])
    B = _blur((rgb[..., 0] - float(T["threshold"])).clamp_(min=0.0), _gauss(20.0, 64))
    E = e + float(T["strength"]) * B[..., None] * _t(T["bleed"])
    D = _t(T["dmax"]) / (1.0 + torch.exp(-_t(T["k"]) * (torch.log10(E.clamp(min=1e-6)) - _t(T["x0"]))))
    if grain:
        for l in range(3):
            n, norm = _grain(h, w, seed, l, _gauss(1.0))
            D[..., l] += float(T["grain"]) * norm * n
    return _scan(D, _t(T["eps"]), _t(T["C"]))


# The differentiable model: theta = wb 3, matrix 9, ev, dmax 3, k 3, x0 3, halation strength, sigma.

def _hal_taps(sigma, dtype):
    x = torch.arange(-64, 65, dtype=dtype, device=DEV)
    g = torch.exp(-x * x / (2.0 * sigma * sigma))
    return g / g.sum()


def _pixel(a, B, dmax, k, x0, strength, dtype):
    """Film RGB of pixels (n, 3) in ACEScg with their halation B (n,)."""
    T = _preset()
    t = {n: _t(T[n]).to(dtype) for n in ("minv", "A", "bleed", "eps", "C")}
    E = (a @ t["minv"].T).clamp(min=0.0) @ t["A"] + strength * B[:, None] * t["bleed"]
    D = dmax / (1.0 + torch.exp(-k * (torch.log10(E.clamp(min=1e-6)) - x0)))
    return torch.exp2(-(D @ t["eps"])) @ t["C"]


def _acescg(x, theta):
    return ((2.0 ** theta[12]) * (theta[0:3] * x)) @ theta[3:12].reshape(3, 3).T


def _model(x, theta, dtype):
    x = x.to(dtype)
    h, w = x.shape[:2]
    a = _acescg(x, theta)
    src = (a[..., 0] - float(_preset()["threshold"])).clamp(min=0.0)
    B = _blur(src, [float(v) for v in _hal_taps(theta[23].double(), torch.float64)]).reshape(-1)
    a = a.reshape(-1, 3)
    out = torch.empty_like(a)
    for i in range(0, h * w, 1 << 20):
        out[i:i + (1 << 20)] = _pixel(a[i:i + (1 << 20)], B[i:i + (1 << 20)], theta[13:16], theta[16:19],
                                      theta[19:22], theta[22], dtype)
    return out.reshape(h, w, 3)


def _fit_exact(case, seed):
    xs, ts = _fit_inputs(case, seed)
    theta = torch.tensor(_f32(synthetic.film_grad_base()), device=DEV)
    out = {"render": _model(xs[0], theta, torch.float64)} if case["render"] else {}
    grad, loss = torch.zeros(24, dtype=torch.float64, device=DEV), 0.0
    scale = float(np.float32(1.0 / (3 * case["images"] * case["w"] * case["h"])))
    for x, t in zip(xs, ts):
        th = theta.clone().requires_grad_(True)
        a = _acescg(x.double(), th)
        src = (a[..., 0] - float(_preset()["threshold"])).clamp(min=0.0)
        B = _blur(src, _hal_taps(th[23], torch.float64))
        # the pixel function in chunks, its gradients to a, B and the curves collected by hand
        af, Bf, tf = a.detach().reshape(-1, 3), B.detach().reshape(-1), t.double().reshape(-1, 3)
        ga, gB = torch.empty_like(af), torch.empty_like(Bf)
        for i in range(0, af.shape[0], 1 << 20):
            sl = slice(i, i + (1 << 20))
            ai, Bi = af[sl].requires_grad_(True), Bf[sl].requires_grad_(True)
            p = theta[13:23].clone().requires_grad_(True)
            r = _pixel(ai, Bi, p[0:3], p[3:6], p[6:9], p[9], torch.float64) - tf[sl]
            l = scale * (r * r).sum()
            ga[sl], gB[sl], gp = torch.autograd.grad(l, (ai, Bi, p))
            grad[13:23] += gp
            loss = loss + l.detach()
        torch.autograd.backward([a, B], [ga.reshape(a.shape), gB.reshape(B.shape)])
        grad += th.grad
        del a, B, src, th
    out["grad"], out["loss"] = grad, loss.reshape(1)
    return out


# The reference stocks used here: 400..700 nm in steps of 20.  Rows: thickness, sensitivity
# (peak, width, height), grain (mean um, sigma), fraction, dye (peak, width), dmax, gamma, capture k.
LAM16 = 400.0 + 20.0 * np.arange(16)
CMF16 = np.array([
    [0.01431, 0.13438, 0.34828, 0.29080, 0.09564, 0.00490, 0.06327, 0.29040, 0.59450, 0.91630, 1.06220, 0.85445,
     0.44790, 0.16490, 0.04677, 0.01136],
    [0.000396, 0.004000, 0.023000, 0.060000, 0.139020, 0.323000, 0.710000, 0.954000, 0.995000, 0.870000, 0.631000,
     0.381000, 0.175000, 0.061000, 0.017000, 0.004100],
    [0.06785, 0.64560, 1.74706, 1.66920, 0.81295, 0.27200, 0.07825, 0.02030, 0.00390, 0.00165, 0.00080, 0.00019,
     0.00002, 0.00000, 0.00000, 0.00000]])
STOCKS = {
    "colorneg200": dict(
        iso=200.0, mask=(0.35, 0.25, 0.05), refl=(680.0, 60.0, 0.08), psf=(3.0, 80.0), dev=8.0, beta=0.35, dirdiff=15.0,
        stack=[("c", 1.0, 0.01), ("e", 4.0, 450.0, 35.0, 1.0, 0.55, 0.3, 0.18, 450.0, 40.0, 2.2, 0.65, 4.2),
               ("g", 2.0, 430.0, 40.0, 1.2), ("e", 5.0, 550.0, 40.0, 1.0, 0.6, 0.32, 0.18, 550.0, 40.0, 2.2, 0.65, 2.1),
               ("e", 6.0, 650.0, 45.0, 1.0, 0.7, 0.35, 0.18, 650.0, 45.0, 2.2, 0.65, 1.35), ("g", 2.0, 650.0, 80.0, 0.3)],
        dir=[[0.02, 0.05, 0.03], [0.05, 0.02, 0.06], [0.03, 0.06, 0.02]]),
    "portra400": dict(
        iso=400.0, mask=(0.32, 0.22, 0.04), refl=(680.0, 60.0, 0.06), psf=(3.0, 70.0), dev=7.0, beta=0.3, dirdiff=16.0,
        stack=[("c", 1.0, 0.01), ("e", 2.5, 450.0, 35.0, 1.0, 0.85, 0.35, 0.16, 450.0, 40.0, 1.1, 0.54, 4.8),
               ("e", 2.5, 450.0, 35.0, 0.8, 0.42, 0.28, 0.2, 450.0, 40.0, 1.1, 0.54, 2.2), ("g", 2.0, 430.0, 40.0, 1.3),
               ("e", 3.0, 550.0, 40.0, 1.0, 0.9, 0.35, 0.16, 550.0, 40.0, 1.1, 0.54, 2.4),
               ("e", 3.0, 550.0, 40.0, 0.8, 0.45, 0.28, 0.2, 550.0, 40.0, 1.1, 0.54, 1.1),
               ("e", 3.5, 650.0, 45.0, 1.0, 0.95, 0.35, 0.16, 650.0, 45.0, 1.1, 0.54, 1.5),
               ("e", 3.5, 650.0, 45.0, 0.8, 0.48, 0.28, 0.2, 650.0, 45.0, 1.1, 0.54, 0.7), ("g", 2.0, 650.0, 80.0, 0.3)],
        dir=[[0.02, 0.01, 0.04, 0.02, 0.03, 0.01], [0.01, 0.01, 0.02, 0.01, 0.02, 0.01],
             [0.04, 0.02, 0.02, 0.01, 0.05, 0.02], [0.02, 0.01, 0.01, 0.01, 0.02, 0.01],
             [0.03, 0.01, 0.05, 0.02, 0.02, 0.01], [0.01, 0.01, 0.02, 0.01, 0.01, 0.01]]),
    "trix400": dict(
        iso=400.0, mask=None, refl=0.01, psf=(3.5, 50.0), dev=6.0, beta=0.35, dirdiff=12.0,
        stack=[("p", 6.0, 0.95, 0.38, 0.22, 1.5, 0.70, 2.2), ("p", 6.0, 0.45, 0.28, 0.24, 1.5, 0.70, 0.9)],
        dir=[[0.03, 0.02], [0.02, 0.02]]),
}


def _reference_stock(name, w):
    """The stock's tables for an image w pixels wide on 35 mm film."""
    sd = STOCKS[name]
    pitch = 36.0 * 1000.0 / w
    trap = np.full(16, 20.0)
    trap[0] = trap[-1] = 10.0
    bump = lambda a, b, c: c * np.exp(-0.5 * ((LAM16 - a) / b) ** 2)  # noqa: E731
    pan = 0.35 + 0.65 * np.maximum(0.0, np.sin(math.pi * (LAM16 - 400.0) / 300.0))
    layers, absorbed, phi = [], [], np.ones(16)
    for row in sd["stack"]:
        if row[0] in "cg":
            phi = phi * np.exp(-(np.full(16, row[2]) if row[0] == "c" else bump(*row[2:5])) * row[1])
            continue
        if row[0] == "p":
            thick, (mean, sig, frac), (dmax, gamma, k) = row[1], row[2:5], row[5:8]
            sens, dye = pan, np.ones(16)
        else:
            thick, (mean, sig, frac), (dmax, gamma, k) = row[1], row[5:8], row[10:13]
            sens, dye = bump(*row[2:5]), bump(row[8], row[9], 1.0)
        after = phi * np.exp(-sens * 2.0 * frac * thick)
        absorbed.append(phi - after)
        phi = after
        layers.append(dict(sens=sens, dye=dye, mean=mean, sig=sig, frac=frac, thick=thick, dmax=dmax, gamma=gamma, k=k))
    basis = np.exp(-0.5 * ((LAM16 - np.array([450.0, 550.0, 650.0])[:, None]) / 40.0) ** 2)
    ap1 = XYZ2AP1 @ CMF16
    minv = np.linalg.inv((ap1 * trap) @ basis.T)
    A = (trap * basis * (LAM16 / 550.0)) @ np.array(absorbed).T / 300.0
    refl = np.full(16, sd["refl"]) if isinstance(sd["refl"], float) else bump(*sd["refl"])
    gains, luts, kappa = [], [], []
    lut_x = -4.0 + np.arange(64) / 63.0 * 12.0
    for L in layers:
        pk = LAM16[int(np.argmax(L["sens"]))]
        wgt = float(np.interp(pk, [450.0, 550.0, 650.0], [0.20, 0.45, 1.0]))
        gains.append(wgt * float((trap * refl * L["sens"]).sum() / (trap * L["sens"]).sum()))
        z = np.linspace(-8.0, 8.0, 65)
        tw = np.full(65, 0.25)
        tw[0] = tw[-1] = 0.125
        s2 = np.exp(2.0 * (math.log(L["mean"]) + L["sig"] * z))
        pdf = np.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi)
        luts.append(np.clip(1.0 - (tw * pdf * np.exp(-L["k"] * s2 * (10.0 ** lut_x)[:, None])).sum(1), 0.0, 1.0))
        r = 0.5 * math.exp(math.log(L["mean"]) + 0.5 * L["sig"] ** 2)
        kappa.append(0.15 / pitch / math.sqrt(L["frac"] * L["thick"] / (4.0 / 3.0 * math.pi * r ** 3)))
    mask = np.zeros(16)
    if sd["mask"]:
        b, g, c = sd["mask"]
        mask = b * bump(450.0, 50.0, 1.0) + g * bump(520.0, 60.0, 0.6) + c
    dmax = np.array([L["dmax"] for L in layers])
    dmin = (ap1 * trap) @ 10.0 ** (-0.4 * dmax.sum() * mask)
    return dict(E=len(layers), minv=minv, A=A, s_local=sd["psf"][0] / pitch, s_wide=sd["psf"][1] / pitch, gains=gains,
                lut_x=lut_x, luts=luts, dmax=dmax, inv_gamma=[1.0 / L["gamma"] for L in layers], masked=bool(sd["mask"]),
                s_dir=sd["dirdiff"] / pitch, dir=np.array(sd["dir"]), s_adj=sd["dev"] / pitch, beta=sd["beta"],
                s_grain=max(3.0 / pitch, 1.0), kappa=kappa, eps=np.array([L["dye"] for L in layers]), mask=mask,
                C=((ap1 * trap) / dmin.max()).T, dmin=dmin / dmin.max(), iso=sd["iso"])


def _reference_scan(rgb, S, seed, grain):
    """Absolute-luminance ACEScg to the scanned negative."""
    E, (h, w) = S["E"], rgb.shape[:2]
    ex = _mat(rgb, S["minv"]).clamp_(min=0.0) @ _t(S["A"])
    P = [ex[..., e].contiguous() for e in range(E)]
    if S["s_local"] >= 1e-3:
        P = [0.82 * p + 0.18 * _blur(p, _gauss(S["s_local"])) for p in P]
    if S["s_wide"] >= 1e-3:
        deep = _blur(P[-1], _gauss(S["s_wide"]))
        P = [p + g * deep if g > 0 else p for p, g in zip(P, S["gains"])]
    x = _t(S["lut_x"])
    M = []
    for e in range(E):
        lp = torch.log10(P[e].clamp(min=1e-300)).clamp_(-4.0, 8.0)
        lo = ((lp + 4.0) * (63.0 / 12.0)).floor().long().clamp_(0, 62)
        t = (lp - x[lo]) / (x[lo + 1] - x[lo])
        fr = _t(S["luts"][e])
        f = (fr[lo] * (1.0 - t) + fr[lo + 1] * t).clamp_(0.0, 1.0)
        P[e] = float(S["dmax"][e]) * f ** S["inv_gamma"][e]
        M.append(0.4 * float(S["dmax"][e]) * (1.0 - f ** S["inv_gamma"][e]) if S["masked"] else None)
    if S["s_dir"] >= 1e-3:
        inh = [_blur(p, _gauss(S["s_dir"])) for p in P]
        P = [P[j] * torch.exp(-sum(float(S["dir"][i, j]) * inh[i] for i in range(E))) for j in range(E)]
    if S["s_adj"] >= 1e-3:
        P = [p + S["beta"] * (p - _blur(p, _gauss(S["s_adj"]))) for p in P]
    if grain:
        for e in range(E):
            dm, k = float(S["dmax"][e]), S["kappa"][e]
            n, norm = _grain(h, w, seed, e, _gauss(S["s_grain"]))
            d = P[e].clamp(0.0, dm)
            taper = (d / (d + 0.02 * dm)).clamp(max=1.0)
            P[e] = (d + k * norm * taper * torch.sqrt((d * (dm - d)).clamp(min=0.0)) * n).clamp(0.0, dm * 1.05)
    if S["masked"]:
        D, eps = torch.stack([*P, sum(M)], -1), np.concatenate([S["eps"], S["mask"][None]])
    else:
        D, eps = torch.stack(P, -1), S["eps"]
    return _scan(D, _t(eps * math.log2(10.0)), _t(S["C"]))


def _invert(rgb, mid, dmin):
    dmin, mid = _t(dmin).clamp(min=1e-6), mid.clamp(min=0.0)
    im_ = (1.0 / (mid / dmin).clamp(1e-6, 1.0 - 1e-6) - 1.0).clamp(min=0.0)
    sh = (im_ * 8.0).clamp(min=1e-6)
    gain = 0.185 / (im_ / (1.0 + im_ / sh)).clamp(min=1e-6)
    inv = (1.0 / (rgb / dmin).clamp(1e-6, 1.0) - 1.0).clamp(min=0.0)
    raw = gain * inv / (1.0 + inv / sh)
    y = (raw @ _t(LUMA)).clamp(min=0.0)[..., None]
    k = 0.55 * (y / 0.02).clamp(max=1.0)
    return (y + k * (raw - y)).clamp(min=0.0)


def _film_exact(case, seed):
    rgb = _image(case["h"], case["w"], seed)
    if case["stock"] == "baseline81":
        return _film81(rgb.double(), _film_seed(seed), case["grain"])
    S = _reference_stock(case["stock"], case["w"])
    out = _reference_scan(rgb.mul_(SUNNY16).double(), S, _film_seed(seed), case["grain"])
    if not case["positive"]:
        return out
    grey = torch.full((32, 32, 3), 0.185 * SUNNY16, dtype=torch.float64, device=DEV)
    mid = _reference_scan(grey, S, 0, case["grain"]).mean((0, 1))
    return _invert(out, mid, S["dmin"])


def _mean3x3(m, pattern, x0, y0):
    """The same-colour mean of the 8 neighbours, the site's own colour keeping its sample."""
    h, w = m.shape
    codes = np.array(["RGB".index(c) for c in pattern]).reshape(6, 6)
    col = torch.as_tensor(codes[np.ix_((np.arange(h) + y0) % 6, (np.arange(w) + x0) % 6)], device=DEV)
    out = torch.empty((h, w, 3), dtype=torch.float64, device=DEV)
    for c in range(3):
        own = (col == c).double()
        s = torch.zeros((h + 2, w + 2), dtype=torch.float64, device=DEV)
        n = torch.zeros_like(s)
        for a in range(3):
            for b in range(3):
                if (a, b) != (1, 1):
                    s[a:a + h, b:b + w] += own * m
                    n[a:a + h, b:b + w] += own
        s, n = s[1:-1, 1:-1], n[1:-1, 1:-1]
        out[..., c] = torch.where(col == c, m, torch.where(n > 0, s / n.clamp(min=1.0), torch.zeros_like(s)))
    return out


def _srgb_encode(v):
    a = v.abs()
    return torch.sign(v) * torch.where(a <= 0.0031308, 12.92 * a, 1.055 * a.clamp(min=1e-12) ** (1 / 2.4) - 0.055)


def _cbrt(v):
    return torch.sign(v) * v.abs() ** (1.0 / 3.0)


def _oklab(v):
    """ACEScg to Oklab."""
    return _mat(_cbrt(_mat(v, OK_M1 @ XYZ2LIN @ AP12XYZ)), OK_M2)


def _from_oklab(v):
    return _mat(_mat(v, OK_M2I) ** 3, XYZ2AP1 @ LIN2XYZ @ OK_M1I)


def _sigmoid(v):
    """Gamut compression, the square sigmoid per channel, chroma scaled by 1 - Y^5 at the compressed
    pixel's hue."""
    ach = v.amax(-1, keepdim=True)
    dist = torch.where(ach == 0, torch.zeros_like(v), (ach - v) / ach.abs().clamp(min=1e-300))
    thr, lim = _t(_f32([0.815, 0.803, 0.88])), _t(_f32([1.147, 1.264, 1.312]))
    p = 1.2
    s = (lim - thr) / ((((1.0 - thr) / (lim - thr)) ** -p - 1.0) ** (1.0 / p))
    d = ((dist - thr) / s).clamp(min=0.0)
    cd = torch.where(dist < thr, dist, thr + s * d / (1.0 + d ** p) ** (1.0 / p))
    gc = torch.where(ach == 0, torch.zeros_like(v), ach - cd * ach.abs())
    hue = _oklab(gc)[..., 1:]
    hue = hue / hue.norm(dim=-1, keepdim=True).clamp(min=1e-300)
    sq = torch.where(gc <= 0, torch.zeros_like(gc), 1.0 / (1.0 + 1.0 / (1.219512 * gc.clamp(min=1e-300))))
    lab = _oklab(sq)
    chroma = lab[..., 1:].norm(dim=-1, keepdim=True) * (1.0 - (sq @ _t(LUMA))[..., None] ** 5)
    return _from_oklab(torch.cat([lab[..., :1], chroma * hue], -1))


def exact(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "develop" and case["sensor"] == "xtrans":
        raw = _raw(h + case["y"] + 5, w + case["x"] + 11, seed, XTRANS, 6)
        m = (raw[case["y"]:case["y"] + h, case["x"]:case["x"] + w].double() - BLACK) / (WHITE - BLACK)
        out = _mat(_mean3x3(m, XTRANS, case["x"], case["y"]) * _t(WB[:3]), XYZ2AP1 @ _camera_matrix())
        return _film81(out, _film_seed(seed), case["grain"]) if case["film"] else out
    if kind == "film":
        return _film_exact(case, seed)
    if kind == "fit":
        return _fit_exact(case, seed)
    if kind == "display":
        v = _image(h, w, seed).double()
        if case["look"] == "filmic":
            v = _mat(_sigmoid(v * 2.0 ** 0.5), XYZ2LIN @ AP12XYZ)
            return torch.where(v <= 0, torch.zeros_like(v), v.clamp(min=1e-300) ** (1.0 / 2.2))
        v = 0.185 * (v.clamp(min=0.0) / 0.185) ** 1.2
        v = _from_oklab(_oklab(v) * _t([1.02, 1.15, 1.15]))
        return _srgb_encode(_mat(v, XYZ2LIN @ AP12XYZ))
    if kind == "preview":
        m, f = _mosaic(h, w, seed, BAYER, 2).double(), case["factor"]
        h2, w2 = h // f, w // f
        site = lambda a, b: m[a::f, b::f][:h2, :w2]  # noqa: E731
        v = torch.stack([site(0, 0), site(1, 0), site(1, 1)], -1)
        v = _film81(_mat(v * _t(WB[:3]), XYZ2AP1 @ _camera_matrix()), _film_seed(seed), True)
        return _srgb_encode(_mat(v, XYZ2LIN @ AP12XYZ))
    return None
