"""Film calls where device memory runs short: the library's working sets come
from the device's current memory pool, so a pool of limited size stands in
for a full device (the driver refuses the allocation; nothing faults).  In a
process of its own, as the pool is the device's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

POOL = """
import numpy as np, torch
import imops_b200 as im
from cuda.bindings import driver as d
x = torch.from_numpy((np.random.default_rng(1).random({shape}) ** 2 * 960).astype(np.float32)).cuda()
small = x[:40, :60].contiguous()
ref = im.FilmStages(stock=2, seed=3, output=0, grain=True).run(x.clone())
ref_small = im.FilmStages(stock=2, seed=3, output=0, grain=True).run(small.clone())
torch.cuda.synchronize()
im.release_working_sets()
props = d.CUmemPoolProps()
props.allocType = d.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
props.location.type = d.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
props.location.id = 0
props.maxSize = {room} << 20
err, pool = d.cuMemPoolCreate(props)
assert err == 0, err
assert d.cuDeviceSetMemPool(0, pool)[0] == 0
def film(v, output=0):
    return im.film_process(v.clone(), stock=2, seed=3, output=output, grain=True)
def check(got, want):
    torch.cuda.synchronize()
    assert torch.equal(got, want)
check(film(small), ref_small)  # the stream holds a small working set from here on
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_grain_beside_the_frame_only_where_there_is_room(gpu):
    """Room for the six-layer frame (120 MiB) but not for planes of the
    grain's own beside it (48 MiB more)."""
    _child(POOL.format(shape=(1300, 1608, 3), room=160) + """
check(film(x), ref)
check(film(x), ref)
err, used = d.cuMemPoolGetAttribute(pool, d.CUmemPool_attribute.CU_MEMPOOL_ATTR_USED_MEM_CURRENT)
assert err == 0 and 119 << 20 < int(used) < 130 << 20, used
check(film(small), ref_small)
""")


def test_calls_after_one_without_room(gpu):
    _child(POOL.format(shape=(1300, 1608, 3), room=64) + """
for output in (1, 0, 1):
    try:
        film(x, output)
        raise SystemExit("no error")
    except im.ImopsError as e:
        assert e.code == 5, e
    check(film(small), ref_small)
""")


@pytest.mark.parametrize("stock,layers", [(0, 1), (6, 2), (1, 3), (2, 6), (4, 7)])
@pytest.mark.parametrize("stage,planes", [("grain", 0), ("develop", 1)])
def test_stages_take_a_plane_a_layer(gpu, stock, layers, stage, planes):
    """The working set of a stage: a plane for each of the stock's layers, and
    one more for the blurs of develop (the block sums and tables are below
    1 MiB here)."""
    import torch
    from cuda.bindings import driver as d

    import imops_b200 as im
    H, W = 1024, 2048
    st = im.FilmStages(stock=stock, seed=3, grain=True)
    v = torch.full((layers, H, W), 0.25, device=gpu)
    torch.cuda.synchronize()
    im.release_working_sets()
    err, pool = d.cuDeviceGetMemPool(0)
    assert err == 0

    def used():
        torch.cuda.synchronize()
        err, n = d.cuMemPoolGetAttribute(pool, d.CUmemPool_attribute.CU_MEMPOOL_ATTR_USED_MEM_CURRENT)
        assert err == 0
        return int(n)

    before = used()
    getattr(st, stage)(v)
    assert used() - before <= (layers + planes) * H * W * 4 + (1 << 20)
    im.release_working_sets()
