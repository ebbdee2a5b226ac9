"""The smallest bakes, whose shadow queues are shorter than the 64 entries a
warp fetches at once, bit for bit against the same texels of a large bake
(paths are keyed by texel and sample, so neighbours change nothing); the
large one against the oracle, to the bounds of the suite's other bakes."""
import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api, scenes

pytestmark = pytest.mark.gpu

CFG = dict(samples=1, bounces=1, seed=8)


@pytest.fixture(scope="module")
def large(gpu_ctx):
    sc = scenes.procedural_room(seed=12, n_boxes=6, res=64, n_point_lights=2)
    pts = api.RasterizeScene(sc, api.RasterConfig(96, 96, 1), ctx=gpu_ctx)
    pts = pts[pts["material_id"] >= 0][::3][:1024]
    assert len(pts) == 1024
    lit = np.zeros(1024, bool)
    for _ in range(2):  # lit texels first (undersides of the boxes see nothing), then the bake of that order
        pts = pts[np.argsort(~lit, kind="stable")]
        out = api.BakeSHLightMap(sc, pts, api.RasterConfig(1024, 1, 1), api.BakeConfig(**CFG), ctx=gpu_ctx)
        lit = np.abs(out.sh_texture.reshape(1024, 27)).max(1) > 0
    return sc, pts, out


def test_large_bake_matches_oracle(large):
    sc, pts, out = large
    ref = O.OracleScene(sc).bake(pts, 1024, 1, 1, **CFG)
    g, r = out.sh_texture.reshape(-1, 27), ref["sh"].reshape(-1, 27)
    assert np.isclose(g, r, rtol=1e-3, atol=1e-5).all(1).mean() >= 0.97
    assert np.linalg.norm(g - r) / np.linalg.norm(r) < 2e-2


@pytest.mark.parametrize("n", [1, 2, 3, 7, 31, 32, 33, 63, 64, 65, 129, 1000])
def test_small_bakes_equal_the_large_one(gpu_ctx, large, n):
    sc, pts, out = large
    got = api.BakeSHLightMap(sc, pts[:n], api.RasterConfig(n, 1, 1), api.BakeConfig(**CFG), ctx=gpu_ctx,
                             with_stats=True)
    assert got.stats.shadow_rays > 0 and np.abs(got.sh_texture).max() > 0
    assert got.sh_texture.tobytes() == out.sh_texture.reshape(-1, 27)[:n].tobytes()
    assert got.environment_visibility_texture.tobytes() == out.environment_visibility_texture.reshape(-1)[:n].tobytes()
