"""Downloads of images into pageable host memory: the bytes of the image at
sizes around the chunks of the threaded copy (below its threshold, one byte's
row more and less than whole chunks, many chunks), from several host threads
at once, after the rings were released, and into pinned memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 4 << 20


def _image(h, w, seed):
    return np.random.default_rng(seed).random((h, w, 3), dtype=np.float32)


@pytest.mark.parametrize("h,w", [(100, 100), (1, 2 * CHUNK // 12), (1, 2 * CHUNK // 12 + 1), (3, CHUNK // 12 + 5),
                                 (512, 2048), (1, 8 * CHUNK // 12), (1, 8 * CHUNK // 12 + 1), (3, 3 * CHUNK // 12 + 5),
                                 (1365, 2049), (2011, 3001)])
def test_round_trip(gpu, h, w):
    import imops_b200 as im
    from imops_b200.pipeline import Image
    x = _image(h, w, seed=h)
    img = Image.from_rgb(x, im.CS_ACESCG)
    assert np.array_equal(img.rgb_f32(), x)
    u8 = np.clip(x, 0.0, 1.0) * np.float32(255.0)
    assert np.array_equal(img.rgb_u8(), u8.astype(np.uint8))
    im.release_working_sets()
    assert np.array_equal(img.rgb_f32(), x)


def test_threads_and_pinned(gpu):
    import ctypes

    import torch

    import imops_b200 as im
    from imops_b200.pipeline import Image
    xs = [_image(1400 + 3 * k, 2000 + k, seed=k) for k in range(6)]  # more at once than there are rings
    imgs = [Image.from_rgb(x, im.CS_ACESCG) for x in xs]
    bad = []

    def run(k):
        for _ in range(3):
            if not np.array_equal(imgs[k].rgb_f32(), xs[k]):
                bad.append(k)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(xs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    pin = torch.empty(xs[0].shape, dtype=torch.float32, pin_memory=True)
    im.check(im.lib().get_image_rgb_f32_c(imgs[0]._h, ctypes.c_void_p(pin.data_ptr()), pin.numel()))
    assert np.array_equal(pin.numpy(), xs[0])
