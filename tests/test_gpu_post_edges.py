"""Downsample and dilation at the edges of their kernels: rows shorter than a
warp, one texel over a block, single rows and columns, scales with and without
a kernel of their own, input rows that the scale leaves over, masks that fill
up before the passes are used, that stay partly empty and that are empty or
full.  Every result is the oracle's, bit for bit, and the allocation-free
dilation's is the same."""
import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from sh_baker_b200 import _capi as A
from sh_baker_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,ch,s", [(64, 48, 27, 2), (99, 33, 27, 3), (100, 34, 27, 3), (37, 9, 27, 4), (5, 5, 27, 5),
                                      (61, 7, 1, 2), (514, 6, 1, 3), (1031, 4, 1, 4), (19, 23, 3, 2), (12, 13, 27, 6)])
def test_downsample(gpu_ctx, w, h, ch, s):
    x = np.random.default_rng(w).normal(size=(h, w, ch)).astype(np.float32)
    got = api._downsample(x, w, h, ch, s, gpu_ctx)
    assert got.tobytes() == O.downsample(x, w, h, ch, s).astype(np.float32).tobytes()


@pytest.mark.parametrize("kind", [A.DILATE_SH9, A.DILATE_F32, A.DILATE_U8])
@pytest.mark.parametrize("w,h,passes,fill", [(1, 1, 3, 0.5), (1, 70, 5, 0.1), (70, 1, 5, 0.1), (31, 33, 1, 0.3),
                                             (32, 8, 2, 0.05), (257, 19, 4, 0.02), (65, 40, 300, 0.01), (40, 40, 3, 0.0),
                                             (40, 40, 3, 1.0), (130, 20, 16, 0.003)])
def test_dilate(gpu_ctx, kind, w, h, passes, fill):
    rng = np.random.default_rng(w * 1000 + h)
    n = w * h
    mask = (rng.random(n) < fill).astype(np.uint8) * rng.integers(1, 256, n).astype(np.uint8)
    if kind == A.DILATE_U8:
        px = rng.integers(0, 256, n).astype(np.uint8)
    else:
        px = rng.normal(size=n * (27 if kind == A.DILATE_SH9 else 1)).astype(np.float32)
    want_px, want_mask = px.copy(), mask.copy()
    O.dilate(kind, w, h, want_px, want_mask, passes)
    got_px, got_mask = px.copy(), mask.copy()
    api.Dilate(w, h, got_px, got_mask, passes, ctx=gpu_ctx)
    assert got_px.tobytes() == want_px.tobytes() and got_mask.tobytes() == want_mask.tobytes()
    d_px, d_mask = torch.from_numpy(px.copy()).cuda(), torch.from_numpy(mask.copy()).cuda()
    torch.cuda.synchronize()
    A.check(gpu_ctx.lib.shb_dilate_noalloc(gpu_ctx.h, kind, w, h, d_px.data_ptr(), d_mask.data_ptr(), passes))
    gpu_ctx.synchronize()
    assert d_px.cpu().numpy().tobytes() == want_px.tobytes() and d_mask.cpu().numpy().tobytes() == want_mask.tobytes()
