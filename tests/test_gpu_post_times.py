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
