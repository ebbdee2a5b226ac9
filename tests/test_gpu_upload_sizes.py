"""Scene uploads around the size of the staging buffer that a context keeps
(32 MiB of page-locked host memory): what fits is laid out whole, more goes
through the buffer's halves in pieces that cut arrays and geometries anywhere.
Most of the vertices belong to no triangle, so that the oracle and the tree
stay small."""
import ctypes as C
import time

import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api
from sh_baker_b200.scene import Geometry, Material, Scene, pack_scene

pytestmark = pytest.mark.gpu

VERTEX = 60  # bytes staged per vertex


def big(sizes, seed=1):
    """Geometries of the given vertex counts, a triangle per 1,000 vertices,
    attributes missing here and there, each with a transform of its own."""
    rng = np.random.default_rng(seed)
    gs = []
    for k, n in enumerate(sizes):
        v = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
        t = max(n // 1000, 1) if n else 0
        idx = rng.integers(0, n, (t, 3)) if n else np.zeros((0, 3))
        if t:
            idx[0], idx[-1] = (0, n // 2, n - 1), (n - 1, n // 3, 0)
        nrm = rng.normal(size=(n, 3)).astype(np.float32)
        tr = np.hstack([np.linalg.qr(rng.normal(size=(3, 3)))[0] * rng.uniform(0.5, 2), rng.uniform(-3, 3, (3, 1))])
        gs.append(Geometry(vertices=v, indices=idx.astype(np.uint32).reshape(-1), transform=tr,
                           normals=nrm if k % 3 else None, texture_uvs=rng.random((n, 2)).astype(np.float32)
                           if k % 2 else None, material_id=0))
    return Scene(gs, [Material()], [])


@pytest.mark.parametrize("sizes", [
    [32 * 2 ** 20 // VERTEX - 10_000],         # a little less than the buffer
    [32 * 2 ** 20 // VERTEX + 10_000],         # a little more
    [3, 0, 700_001, 0, 0, 900_000, 1, 5, 0],
    [1_398_101, 1, 1_500_000],                 # the positions that a half holds, and one more
    [n for k in range(2000) for n in (k % 7, 1500)],
])
def test_contents(gpu_ctx, sizes):
    sc = big(sizes)
    rng = np.random.default_rng(2)
    rays = np.empty((20_000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-8, 8, (20_000, 3))
    rays[:, 3:6] = rng.uniform(-3, 3, (20_000, 3)) - rays[:, 0:3]
    rays[:, 6], rays[:, 7] = 0.0, np.inf
    got = api.FindOcclusion(sc, rays, ctx=gpu_ctx)
    want = O.OracleScene(sc).find_occlusion(rays)
    assert (want["hit"] == 1).sum() > 100
    same = (got["hit"] == want["hit"]) & (got["prim_id"] == want["prim_id"])
    assert (~same).sum() <= 10  # 5 in 10,000 graze an edge
    for name in ("t", "position", "normal", "uv", "material_id"):
        assert np.array_equal(got[name][same], want[name][same]), name


def test_time_grows_with_the_bytes(gpu_ctx):
    # twice the bytes across the buffer's size: three times the time is
    # generous; in plain memory of its own the larger one took about ten times
    ms = []
    for n in (450_000, 900_000, 1_800_000):
        desc, keep = pack_scene(big([n]))
        ts = []
        for _ in range(6):
            h = C.c_void_p()
            t = time.perf_counter()
            assert gpu_ctx.lib.shb_scene_upload(gpu_ctx.h, C.byref(desc), C.byref(h)) == 0
            ts.append(time.perf_counter() - t)
            gpu_ctx.lib.shb_scene_destroy(h)
        ms.append(min(ts) * 1e3)
    assert ms[1] < 3 * ms[0] and ms[2] < 3 * ms[1], ms


def locked():
    """Bytes of shared memory this process holds, as which the driver's
    page-locked host memory counts."""
    return int(next(x for x in open("/proc/self/status") if x.startswith("RssShmem:")).split()[1]) << 10


@pytest.mark.parametrize("vertices,kept", [(1_000, 2 << 20), (300_000, 300_000 * VERTEX * 9 // 8 + (1 << 20)),
                                           (900_000, 32 << 20), (1_800_000, 32 << 20)])
def test_first_upload_locks_no_more_than_it_needs(vertices, kept):
    # A context's first upload waits until its staging buffer is locked, about
    # 0.6 ms per MiB: what the upload needs and an eighth, at most 32 MiB (the
    # driver rounds to 2 MiB).
    from sh_baker_b200 import Context
    desc, keep = pack_scene(big([vertices]))
    ctx = Context()
    before = locked()
    h = C.c_void_p()
    assert ctx.lib.shb_scene_upload(ctx.h, C.byref(desc), C.byref(h)) == 0
    ctx.lib.shb_scene_destroy(h)
    grown = locked() - before
    ctx.close()
    assert 0 < grown <= kept + (2 << 20)
    assert locked() < before + grown  # given back with the context
