"""A table with a negative light (a fill that takes light away), whose running
sums may fall: the pick still searches them, and evaluates no light again.
One light of 24 made slightly negative changes no work, at most the sums'
search; the bound of a third more shading time leaves room for that (a second
light loop per pick took three quarters more)."""
import numpy as np
import pytest

from sh_baker_b200 import api, scenes
from sh_baker_b200.scene import POINT, Light

pytestmark = pytest.mark.gpu


def shading_ms(ctx, last):
    sc = scenes.procedural_room(seed=3, n_boxes=60, res=256, n_point_lights=0)
    rng = np.random.default_rng(4)
    sc.lights = [Light(type=POINT, position=tuple(float(x) for x in rng.uniform((-4, 1.5, -4), (4, 2.8, 4))),
                       intensity=float(rng.uniform(5, 20))) for _ in range(24)]
    sc.lights[-1].intensity = last
    ds = api.DeviceScene(ctx, sc)
    rc = api.RasterConfig(512, 512, 1)
    g = api.rasterize_to_device(ds, rc)
    times = [api.BakeSHLightMap(ds, g, rc, api.BakeConfig(samples=64, bounces=3, seed=5), ctx=ctx,
                                with_stats=True).stats.shade_kernel_ms for _ in range(6)]
    return min(times)


def test_negative_light_costs_no_second_loop():
    from sh_baker_b200 import Context
    ctx = Context(profiling=True)
    assert shading_ms(ctx, -0.01) < 4.0 / 3.0 * shading_ms(ctx, 0.01)
    ctx.close()
