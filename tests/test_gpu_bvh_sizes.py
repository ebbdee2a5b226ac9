"""The BVH builder at the sizes where its phases hand over: a leaf, the
eight-lane subtrees (up to 8 triangles), the block-wide ones (up to 512) and
the levels above, with coincident, flat and clustered triangles, whose splits
fall to the median or peel off few triangles at a time.  Closest hits are
compared with the oracle's, which has a tree of its own, and a rebuild gives
the same hits and tree."""
import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api
from sh_baker_b200.scene import Geometry, Material, Scene

pytestmark = pytest.mark.gpu


def soup(n, kind):
    rng = np.random.default_rng(n)
    v = rng.uniform(-1, 1, (n, 3, 3)) * 0.3 + rng.uniform(-2, 2, (n, 1, 3))
    if kind == "same":
        v[:] = v[0]
    elif kind == "flat":
        v[:, :, 2] = 0.25
    elif kind == "spread":  # sizes and places over many orders of magnitude
        v *= np.exp(rng.uniform(-10, 0, (n, 1, 1)))
    return Scene([Geometry(vertices=v.reshape(-1, 3).astype(np.float32), indices=np.arange(3 * n, dtype=np.uint32),
                           material_id=0)], [Material()], [])


@pytest.mark.parametrize("n,kind", [(n, "random") for n in (1, 2, 3, 4, 8, 9, 16, 17, 255, 257, 511, 512, 513, 1025, 3000)]
                         + [(9, "same"), (513, "same"), (2000, "same"), (600, "flat"), (700, "spread"), (4000, "spread")])
def test_sizes(gpu_ctx, n, kind):
    sc = soup(n, kind)
    rng = np.random.default_rng(1)
    rays = np.empty((4000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-3, 3, (4000, 3))
    verts = sc.geometries[0].vertices.reshape(-1, 3, 3).mean(1)
    rays[:, 3:6] = verts[rng.integers(0, n, 4000)] + rng.normal(size=(4000, 3)) * 0.05 - rays[:, 0:3]
    rays[:, 6], rays[:, 7] = 0.001, np.inf
    ds = api.DeviceScene(gpu_ctx, sc)
    info = ds.bvh_info()
    assert info["triangles"] == n and 1 <= info["wide_nodes"] <= max(n, 1) and 1 <= info["depth"] <= 64
    got = api.FindOcclusion(ds, rays, ctx=gpu_ctx)
    want = O.OracleScene(sc).find_occlusion(rays)
    same = got["hit"] == want["hit"]
    assert (~same).sum() <= 2  # rays that graze an edge: the box tests do not round alike
    both = same & (got["hit"] == 1)
    np.testing.assert_allclose(got["t"][both], want["t"][both], rtol=1e-5, atol=1e-6)
    if kind not in ("same", "flat"):  # coplanar triangles that overlap are hit at one distance: any of them is right
        assert (got["prim_id"][both] != want["prim_id"][both]).sum() <= 2
    ds.rebuild_bvh()
    assert ds.bvh_info() == info
    assert api.FindOcclusion(ds, rays, ctx=gpu_ctx).tobytes() == got.tobytes()
