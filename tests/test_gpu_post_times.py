"""Post-processing times compared with one another on the same device: what
reads twice the bytes takes about twice the time, whatever the scale or the
shape of the image.  The bounds leave a factor of one and a half or more."""
import pytest
import torch

from sh_baker_b200 import Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def timed():
    ctx = Context()
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)

    def us(call, n=10):
        for _ in range(3):
            call(ctx)
        torch.cuda.synchronize()
        best = 1e30
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            for _ in range(n):
                call(ctx)
            b.record(stream)
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) / n * 1e3)
        return best
    yield us
    ctx.close()


def downsample_us(timed, w, h, ch, s):
    x = torch.rand(w * s * h * s * ch, device="cuda")
    y = torch.empty(w * h * ch, device="cuda")
    return timed(lambda c: c.lib.shb_downsample(c.h, x.data_ptr(), w * s, h * s, ch, s, y.data_ptr(), 1))


def test_sh_downsample_scales(timed):
    # 5, 10 and 17 floats moved per output float; scale 2 took 1.6 times scale
    # 3's time and scale 4 four times
    t2, t3, t4 = (downsample_us(timed, 1000, 1000, 27, s) for s in (2, 3, 4))
    assert t2 < 0.8 * t3 and t4 < 2.5 * t3, (t2, t3, t4)


@pytest.mark.parametrize("ch", [1, 27])
@pytest.mark.parametrize("w", [1, 3, 17])
def test_thin_images_downsample(timed, w, ch):
    # the square's texels in narrow rows; with a block per row one column took
    # four (27 channels) to eleven times the square's time
    n = 1 << 19 if ch == 1 else 1 << 17
    side = int(n ** 0.5)
    square, thin = downsample_us(timed, side, side, ch, 2), downsample_us(timed, w, n // w, ch, 2)
    assert thin < 2.5 * square + 5.0, (square, thin)


@pytest.mark.parametrize("w", [1, 3, 17])
def test_thin_masks(timed, w):
    n = 1 << 20
    m = torch.ones(n * 4, dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    square, thin = (timed(lambda c: c.lib.shb_downsample_validity_mask(c.h, m.data_ptr(), a, n // a, 2, out.data_ptr(), 1))
                    for a in (1024, w))
    assert thin < 2.5 * square + 5.0, (square, thin)


@pytest.mark.parametrize("ch", [1, 5, 27])
def test_short_rows_match_oracle(ch):
    # several rows a block, up to and beyond its 256 elements
    import numpy as np

    from oracle import pyoracle as O
    from sh_baker_b200 import api
    ctx = Context()
    rng = np.random.default_rng(ch)
    for w, h in ((1, 4001), (2, 777), (3, 1000), (9, 95), (10, 33), (51, 40), (52, 41), (255, 9), (257, 5), (600, 3)):
        for s in (2, 3, 4, 5):
            x = rng.normal(size=(h * s + s // 2, w * s + 1, ch)).astype(np.float32)
            got = api._downsample(x, x.shape[1], x.shape[0], ch, s, ctx)
            assert got.tobytes() == O.downsample(x, x.shape[1], x.shape[0], ch, s).astype(np.float32).tobytes(), (w, h, s)
        m = (rng.random((h * 3, w * 3)) < 0.1).astype(np.uint8)
        want = m.reshape(h, 3, w, 3).max(axis=(1, 3))
        assert np.array_equal(api.DownsampleValidityMask(m, w, h, 3, ctx=ctx).reshape(h, w), want)
    ctx.close()
