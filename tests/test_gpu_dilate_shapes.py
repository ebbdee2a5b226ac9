"""Dilation at the sizes and shapes where its kernels change: up to 8,192
texels of SH9 and 160,000 of one channel a thread per float, above that tiles
whose width follows narrow and flat images.  Compared with the oracle's passes
bit for bit, and in time: one column or row, and a small image of isolated
texels, take no more than a small multiple of the ordinary case."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from sh_baker_b200 import Context, api

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 8192), (1, 8193), (8193, 1), (2, 5000), (5000, 2), (3, 2731), (4, 9001), (5, 1700), (7, 1171), (9, 911),
          (33, 257), (64, 128), (65, 127), (91, 91), (130, 131), (3001, 3), (3000, 4), (40, 8), (8, 40)]
SHAPES_1 = [(400, 400), (401, 400), (1, 160_001), (160_001, 1), (2, 81_000), (81_000, 2), (17, 9500), (500, 333)]


@pytest.mark.parametrize("kind", ["sh", "f32", "u8"])
@pytest.mark.parametrize("density", [0.002, 0.05, 0.7])
def test_shapes_match_oracle(gpu_ctx, kind, density):
    for w, h in SHAPES + (SHAPES_1 if kind != "sh" else []):
        rng = np.random.default_rng(w * 7 + h)
        n = w * h
        mask = (rng.random(n) < density).astype(np.uint8) * 3
        mask[rng.integers(0, n)] = 1
        px = (rng.integers(0, 256, n).astype(np.uint8) if kind == "u8" else
              rng.normal(size=n * (27 if kind == "sh" else 1)).astype(np.float32))
        for passes in (1, 3, 6):
            g, gm, r, rm = px.copy(), mask.copy(), px.copy(), mask.copy()
            api.Dilate(w, h, g, gm, passes, ctx=gpu_ctx)
            O.lib().oracle_dilate({"sh": 0, "f32": 1, "u8": 2}[kind], w, h, r.ctypes.data, rm.ctypes.data, passes)
            assert gm.tobytes() == rm.tobytes() and g.tobytes() == r.tobytes(), (w, h, passes)


@pytest.fixture(scope="module")
def timed():
    ctx = Context()
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)

    def us(w, h, kind, density, passes, n=10):
        ch = 27 if kind == 0 else 1
        torch.manual_seed(1)
        m0 = (torch.rand(w * h, device="cuda") < density).to(torch.uint8)
        m, px = m0.clone(), torch.rand(w * h * ch, device="cuda")
        torch.cuda.synchronize()

        def call():
            m.copy_(m0)
            assert ctx.lib.shb_dilate(ctx.h, kind, w, h, C.c_void_p(px.data_ptr()), C.c_void_p(m.data_ptr()), passes, 1) == 0
        best = 1e30
        with torch.cuda.stream(stream):
            for _ in range(6):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                for _ in range(n):
                    call()
                b.record(stream)
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b) / n * 1e3)
        return best
    yield us
    ctx.close()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("w", [1, 3])
def test_time_of_narrow_images(timed, kind, w):
    # nothing to fill: a pass reads the labels.  With 64 x 16 tiles one column
    # took nine (one float) and fourteen (SH9) times the square's time
    n = 1 << 20
    assert timed(w, n // w, kind, 0.0, 1) < 2.5 * timed(1024, 1024, kind, 0.0, 1) + 5.0


def test_time_of_small_images(timed):
    # 64^2 SH9 texels, two in a hundred valid: 4 passes fill most of them.  The
    # bare launches of an empty mask take a third of what the tiles took
    assert timed(64, 64, 0, 0.02, 4) < 2.0 * timed(64, 64, 0, 0.0, 4)
