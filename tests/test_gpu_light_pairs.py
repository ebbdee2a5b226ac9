"""Next-event estimation over light tables at the edges of its code: lights
weighed in pairs and left over, coloured and grey, area lights of constant
and of textured emission, tables beyond the cached (32) and the staged (64)
size, samples of one texel that fill a warp, part of one, or straddle two,
and several light samples.  Each bake is compared with the oracle's on the
same counter stream: both evaluate the same float expressions, so texels
agree to rounding except where a 1-ulp difference of a transcendental moves a
path (the bounds of the suite's other oracle bakes).

The pick searches the cached running sums, or, for larger tables and where a
negative light lets the sums fall, evaluates the lights again in order.
Lights of zero intensity at the end of the table weigh nothing and change no
draw, so a table padded past the cache must give the same bits."""
import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api, scenes
from sh_baker_b200.scene import DIRECTIONAL, POINT, SPOT, Light, Material, Texture

pytestmark = pytest.mark.gpu


def lit_room(points, areas, textured, extra, seed=5):
    sc = scenes.procedural_room(seed=seed, n_boxes=10, res=48, n_point_lights=0)
    rng = np.random.default_rng(seed)
    for i in range(points):
        color = (1.0, 1.0, 1.0) if i % 3 else tuple(float(x) for x in rng.uniform(0.2, 1.0, 3))
        sc.lights.append(Light(type=POINT, position=tuple(float(x) for x in rng.uniform((-4, 1.5, -4), (4, 2.8, 4))),
                               color=color, intensity=float(rng.uniform(5, 30))))
    for i in range(areas):
        if textured and i == textured - 1:
            px = rng.integers(0, 256, (4, 4, 3)).astype(np.uint8)
            albedo = Texture(4, 4, 3, px.reshape(-1))
        else:
            albedo = Texture(1, 1, 3, rng.integers(100, 256, 3).astype(np.uint8))
        sc.materials.append(Material(name=f"e{i}", albedo=albedo, emission_intensity=float(rng.uniform(1, 5))))
        sc.geometries[1 + i].material_id = len(sc.materials) - 1
    scenes.mark_area_lights(sc)
    if extra == "spot":
        sc.lights.insert(1, Light(type=SPOT, position=(0.0, 2.9, 0.0), direction=(0.0, -1.0, 0.0), intensity=30.0,
                                  cos_inner_cone=0.9, cos_outer_cone=0.6))
    if extra == "negative":
        sc.lights.append(Light(type=POINT, position=(1.0, 2.0, 1.0), intensity=-2.0))
        sc.lights.append(Light(type=DIRECTIONAL, direction=(0.0, -1.0, 0.0), intensity=1.0))
    return sc


@pytest.mark.parametrize("points,areas,textured,extra,spp,nls", [
    (1, 0, 0, None, 32, 1), (2, 0, 0, None, 16, 1), (3, 0, 0, "spot", 32, 2), (4, 1, 0, None, 33, 1),
    (2, 2, 0, None, 48, 1), (3, 5, 0, "spot", 32, 2), (0, 4, 1, None, 32, 1), (1, 5, 3, None, 24, 1),
    (31, 0, 0, None, 32, 1), (32, 0, 0, None, 32, 1), (34, 2, 0, None, 32, 1), (66, 0, 0, None, 32, 1),
])
def test_light_tables_match_oracle(gpu_ctx, points, areas, textured, extra, spp, nls):
    sc = lit_room(points, areas, textured, extra)
    osc = O.OracleScene(sc)
    pts = osc.rasterize(48, 48, 1)
    ref = osc.bake(pts, 48, 48, 1, samples=spp, bounces=2, seed=31, num_light_samples=nls)
    got = api.BakeSHLightMap(sc, pts, api.RasterConfig(48, 48, 1),
                             api.BakeConfig(samples=spp, bounces=2, seed=31, num_light_samples=nls), ctx=gpu_ctx)
    valid = (pts["material_id"] >= 0).reshape(48, 48)
    g, r = got.sh_texture[valid].reshape(-1, 27), ref["sh"][valid].reshape(-1, 27)
    close = np.isclose(g, r, rtol=1e-3, atol=1e-5).all(axis=1)
    assert close.mean() >= 0.97, close.mean()
    assert np.linalg.norm(g - r) / max(np.linalg.norm(r), 1e-12) < 2e-2


@pytest.mark.parametrize("points,areas,textured,extra,nls", [
    (1, 0, 0, None, 1), (4, 0, 0, "spot", 2), (5, 0, 0, "negative", 1), (2, 3, 0, "negative", 2), (3, 5, 2, None, 1),
    (20, 8, 0, None, 1),
])
def test_pick_from_sums_equals_scan(gpu_ctx, points, areas, textured, extra, nls):
    out = []
    for pad in (0, 40):
        sc = lit_room(points, areas, textured, extra)
        sc.lights += [Light(type=POINT, position=(0.0, 2.0, 0.0), intensity=0.0) for _ in range(pad)]
        ds = api.DeviceScene(gpu_ctx, sc)
        rc = api.RasterConfig(48, 48, 1)
        pts = api.RasterizeScene(ds, rc, ctx=gpu_ctx)
        out.append(api.BakeSHLightMap(ds, pts, rc, api.BakeConfig(samples=32, bounces=2, seed=8, num_light_samples=nls),
                                      ctx=gpu_ctx).sh_texture)
    assert np.abs(out[0]).max() > 0 and out[0].tobytes() == out[1].tobytes()
