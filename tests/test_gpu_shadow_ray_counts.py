"""Light queries (BakeStats.shadow_rays) and any-hit rays traced
(Context.shadow_rays_traced): equal where no two samples can share a ray, and
otherwise one ray per light that the samples of a texel in one warp query."""
import numpy as np
import pytest
import torch

from sh_baker_b200 import AREA, Context, api, scenes
from sh_baker_b200.scene import POINT, Light

pytestmark = pytest.mark.gpu


def bake(ctx, sc, res, **cfg):
    rc = api.RasterConfig(res, res, 1)
    ds = api.DeviceScene(ctx, sc)
    g = api.rasterize_to_device(ds, rc)
    before = ctx.shadow_rays_traced()
    st = api.BakeSHLightMap(ds, g, rc, api.BakeConfig(seed=5, **cfg), ctx=ctx, with_stats=True).stats
    return ctx.shadow_rays_traced() - before, st


def test_shared_rays_of_a_texel(gpu_ctx):
    sc = scenes.unit_quad()  # nothing to hit: texel queries only
    sc.lights = [Light(type=POINT, position=(0.0, 1.0, 0.0), intensity=10.0)]
    for spp, rays in ((1, 1), (32, 1), (64, 2)):  # every sample queries the one light; a warp holds 32
        traced, st = bake(gpu_ctx, sc, 32, samples=spp, bounces=1)
        assert st.shadow_rays == 1024 * spp and traced == 1024 * rays


@pytest.mark.parametrize("area", [False, True])
def test_one_sample_shares_nothing(gpu_ctx, area):
    sc = scenes.procedural_room(seed=4, n_boxes=10, res=32, n_point_lights=4)
    if area:  # area lights sample a point per path
        sc.lights = []
        sc.materials[sc.geometries[1].material_id].emission_intensity = 5.0
        scenes.mark_area_lights(sc)
        assert {light.type for light in sc.lights} == {AREA}
    traced, st = bake(gpu_ctx, sc, 32, samples=32 if area else 1, bounces=2)
    assert traced == st.shadow_rays > 0


def test_counts_add_up_over_calls():
    ctx = Context()
    assert ctx.shadow_rays_traced() == 0
    sc = scenes.procedural_room(seed=4, n_boxes=10, res=32, n_point_lights=4)
    a, st = bake(ctx, sc, 32, samples=16, bounces=1)
    b, _ = bake(ctx, sc, 32, samples=16, bounces=1)
    assert 0 < a < st.shadow_rays and a == b and ctx.shadow_rays_traced() == 2 * a
    ds = api.DeviceScene(ctx, sc)
    rc = api.RasterConfig(32, 32, 1)
    bakes = [api.BatchBake(ds, api.rasterize_to_device(ds, rc), rc, api.BakeConfig(samples=16, bounces=1, seed=5))] * 3
    torch.cuda.synchronize()
    _, st3 = api.bake_batch(ctx, bakes, wave_paths=1 << 12)
    assert ctx.shadow_rays_traced() == 5 * a and st3.shadow_rays == 3 * st.shadow_rays
    ctx.close()
