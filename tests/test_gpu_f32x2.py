"""The packed operations that weigh two lights at once (f32x2.cuh) against the
scalar ones, bit for bit: the light picks rest on their rounding alike.
Compiled with the light kernels' own flags, because what they rely on is the
assembler's doing: a packed product and a packed sum must not be contracted
into one multiply-add.  Quotients are tested over the ranges that the pairs
are held to, with mantissas at and next to powers of two among them."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from sh_baker_b200 import build as B

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
N = 1 << 22


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = tmp_path_factory.mktemp("f32x2") / "f32x2_probe.so"
    subprocess.run([B.nvcc(), *B.ARCH, *B.COMMON, *B.SOURCES["shade.cu"], "-shared", "-I", str(B.CSRC), "-I",
                    str(ROOT / "include"), str(ROOT / "tests" / "cpp" / "f32x2_probe.cu"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def values(rng, lo, hi, n=N):
    """Floats of both signs with exponents spread over lo .. hi, a quarter of
    them with a mantissa within 3 of a power of two."""
    m = rng.integers(0, 1 << 23, n)
    edge = rng.random(n) < 0.25
    m[edge] = rng.integers(-3, 4, edge.sum()) % (1 << 23)
    e = rng.integers(int(np.floor(np.log2(lo))), int(np.floor(np.log2(hi))) + 1, n)
    v = np.clip(np.ldexp(1.0 + m * 2.0 ** -23, e), lo, hi).astype(np.float32)
    return v * rng.choice(np.float32([1, -1]), n)


def run(probe, a, b, c):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (a, b, c)]
    out = torch.empty(6 * N, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert probe.f32x2_probe(*[C.c_void_p(x.data_ptr()) for x in t], C.c_int64(N), C.c_void_p(out.data_ptr())) == 0
    return out.cpu().numpy().view(np.uint32).reshape(6, N)


def limits(probe):
    r = (C.c_float * 4)()
    probe.f32x2_range(r)
    return [float(x) for x in r]


def test_quotients(probe):
    dim, bright, near, far = limits(probe)
    rng = np.random.default_rng(1)
    d = np.abs(values(rng, near, far))
    for a, b in [(values(rng, dim, bright), d * d),                # an emission by the squared distance
                 (values(rng, dim, dim * 4), np.clip(d * d, far * far / 16, far * far)),
                 (values(rng, bright / 4, bright), np.clip(d * d, near * near, near * near * 16)),
                 # a component of the way by the distance, down to 2^-96
                 (d * np.clip(values(rng, 2.0 ** -60, 1.0), -1, 1), d),
                 (values(rng, 2.0 ** -96, 2.0 ** -90), np.maximum(d, np.float32(2.0) ** -30))]:
        got, want = run(probe, a, b.astype(np.float32), a)[:2]
        assert np.isfinite(want.view(np.float32)).all()
        assert np.array_equal(got, want), int((got != want).sum())


def test_no_quotient_of_the_range_is_subnormal(probe):
    # below 2^-126 a quotient half way between two floats may round either way
    dim, bright, near, far = limits(probe)
    rng = np.random.default_rng(3)
    b = np.ldexp(rng.integers(1, 1 << 11, N) * 2.0 + 1.0, rng.integers(30, 49, N))
    a = b * (rng.integers(1, 1 << 10, N) * 2.0 + 1.0) * 2.0 ** -150  # exact in 24 bits
    inside = (a >= dim) & (a <= bright) & (b >= near * near) & (b <= far * far)
    if inside.any():
        a, b = (np.resize(x[inside], N).astype(np.float32) for x in (a, b))
        got, want = run(probe, a, b, a)[:2]
        assert np.array_equal(got, want), int((got != want).sum())
    assert dim / far ** 2 >= 2.0 ** -126 and bright / near ** 2 < 2.0 ** 127
    assert dim * 2.0 ** -47 >= 2.0 ** -149  # residuals are multiples of this


def test_products_are_rounded_by_themselves(probe):
    rng = np.random.default_rng(2)
    a, b = values(rng, 2.0 ** -20, 2.0 ** 20), values(rng, 2.0 ** -20, 2.0 ** 20)
    c = -(a * b) * rng.choice(np.float32([1, 1, 0.5, 1 + 2.0 ** -23]), N)  # sums that show the product's rounding
    a[:8], b[:8] = [0.0, -0.0, 0.0, -0.0, 3.0, -3.0, 0.0, 5.0], [2.0, 2.0, -2.0, -2.0, 0.0, 0.0, -0.0, -0.0]
    out = run(probe, a, b, c)
    assert np.array_equal(out[2], out[3]) and np.array_equal(out[4], out[5])
