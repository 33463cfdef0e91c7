"""Film calls of different callers stay independent: what one stream has queued
holds up no film on another, and a film that is being captured into a graph
does not disturb one that runs.  In a process of its own, with a hardware
queue for every stream, so that streams that share a queue hold up nothing
here."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
import numpy as np, torch
import imops_b200 as im
rng = np.random.default_rng(1)
frame = lambda h, w: torch.from_numpy((rng.random((h, w, 3)) ** 2 * 960).astype(np.float32)).cuda()
xa, xb = frame(1200, 1600), frame(700, 1000)
A, B = torch.cuda.Stream(), torch.cuda.Stream()
kinds = [dict(stock=1, seed=2, output=1), dict(stock=2, seed=2, output=0), dict(stock=1, seed=2, output=0),
         dict(stock=im.STOCK_BASELINE81)]
def film(x, stream, kind):
    with torch.cuda.stream(stream):
        return im.film_process(x, **kinds[kind])
ref = [[film(x.clone(), s, k) for x, s in ((xa, A), (xb, B))] for k in range(len(kinds))]  # the working sets exist from here on
torch.cuda.synchronize()
"""


def _child(code):
    env = dict(os.environ, CUDA_DEVICE_MAX_CONNECTIONS="32")
    r = subprocess.run([sys.executable, "-c", SETUP + code], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_a_busy_stream_holds_up_no_other(gpu):
    """Half a second of other work is queued on A before its film (a positive,
    with its mid-grey patch; negatives, with their grain beside the frame; the
    preset): B's film is done before that work is."""
    _child("""
for a in range(4):
    for b in range(4):
        va, vb = xa.clone(), xb.clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(A):
            torch.cuda._sleep(1_000_000_000)
        slept = A.record_event()
        film(va, A, a)
        film(vb, B, b)
        B.synchronize()
        assert not slept.query(), f"film {b} on B waited for A (film {a})"
        A.synchronize()
        assert torch.equal(va, ref[a][0]) and torch.equal(vb, ref[b][1])
""")


def test_a_film_runs_while_another_is_captured(gpu):
    _child("""
for a, b in [(0, 0), (0, 1), (1, 0), (1, 2), (3, 0), (0, 3), (3, 3)]:
    va, vb = xa.clone(), xb.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=A, capture_error_mode="relaxed"):
        film(va, A, a)
        film(vb, B, b)
        B.synchronize()
    assert torch.equal(vb, ref[b][1]) and torch.equal(va, xa)
    for _ in range(2):
        va.copy_(xa)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(va, ref[a][0])
    del g
""")
