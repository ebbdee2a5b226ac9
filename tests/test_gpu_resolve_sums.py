"""The resolve kernel's lane sums at sample counts around the warp's width,
and its zero paths: a path without radiance adds zeros, unless its direction
is so long that a product of its components is infinite (0 * inf)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("scale", [1.0, 9e3, 1.1e4, 1e18])
def test_paths_without_radiance(gpu_ctx, scale, spp):
    sc = scenes.unit_quad()
    sc.lights = []
    rc = api.RasterConfig(8, 8, 1)
    pts = api.RasterizeScene(sc, rc, ctx=gpu_ctx)
    pts["normal"] *= np.float32(scale)
    pts["tangent"][..., :3] *= np.float32(scale)
    res = api.BakeSHLightMap(sc, pts, rc, api.BakeConfig(samples=spp, bounces=1, seed=4), ctx=gpu_ctx)
    sh = res.sh_texture.reshape(64, 9, 3)
    # at 1e18 the bitangent is 1e36 long: the coefficients with its axis twice,
    # or once beside another, overflow
    axis = int(np.abs(np.cross(pts["normal"], pts["tangent"][..., :3])).reshape(-1, 3)[0].argmax())
    over = [[4, 7, 8], [4, 5, 8], [5, 6, 7]][axis] if scale == 1e18 else []
    assert np.isnan(sh[:, over]).all()
    assert (np.delete(sh, over, axis=1) == 0).all()
    assert (res.environment_visibility_texture == 1).all()


@pytest.mark.parametrize("spp", [1, 3, 31, 32, 33, 65])
def test_sums_against_the_oracle(gpu_ctx, spp):
    sc = scenes.procedural_room(seed=9, n_boxes=6, res=16, n_point_lights=2)
    rc = api.RasterConfig(16, 16, 1)
    pts = api.RasterizeScene(sc, rc, ctx=gpu_ctx)
    res = api.BakeSHLightMap(sc, pts, rc, api.BakeConfig(samples=spp, bounces=2, seed=21), ctx=gpu_ctx)
    ref = O.OracleScene(sc).bake(pts.reshape(-1), 16, 16, 1, samples=spp, bounces=2, seed=21)
    valid = pts.reshape(16, 16)["material_id"] >= 0
    g, r = res.sh_texture[valid].reshape(-1, 27), ref["sh"][valid].reshape(-1, 27)
    # a path that grazes an edge may part from the oracle's; the other texels
    # differ by the rounding of at most 65 terms
    close = np.isclose(g, r, rtol=2e-4, atol=2e-5 * max(1.0, float(np.abs(r).max()))).all(1)
    assert close.mean() > 0.95
    np.testing.assert_allclose(res.environment_visibility_texture, ref["env"], atol=2.0 / spp + 1e-6)
