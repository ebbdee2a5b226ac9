"""Next-event estimation of a warp whose lanes disagree on a pair of area
lights: the lights reach beyond 2^30 from the texel, so that some lanes'
samples lie within the range in which two lights are weighed at once and some
do not.  The warp must still meet each point and spot light together, whose
weights it shares.  A table padded with lights of zero intensity beyond 32
entries is evaluated lane by lane, without sharing, and must give the same
bits; the lights' intensities are such that the far lights' weights reach the
sums' last bits."""
import numpy as np
import pytest

from sh_baker_b200 import api, scenes
from sh_baker_b200.scene import POINT, SPOT, Geometry, Light, Material, Texture

pytestmark = pytest.mark.gpu

FAR = 1.5 * 2.0 ** 30


def far_lit_room(areas):
    sc = scenes.procedural_room(seed=5, n_boxes=10, res=48, n_point_lights=0)
    rng = np.random.default_rng(7)
    sc.lights = []
    for k in range(areas):
        v = np.float32([[0, 20 + k, 0], [FAR, 20 + k, 0], [0, 20 + k, FAR]])
        sc.materials.append(Material(name=f"far{k}", albedo=Texture(1, 1, 3, np.uint8([255, 255, 255])),
                                     emission_intensity=2.0 ** 29))
        sc.geometries.append(Geometry(vertices=v, indices=np.uint32([0, 1, 2]), normals=np.float32([[0, -1, 0]] * 3),
                                      tangents=np.float32([[1, 0, 0, 1]] * 3), lightmap_uvs=np.full((3, 2), -1, np.float32),
                                      texture_uvs=np.zeros((3, 2), np.float32), material_id=len(sc.materials) - 1))
    scenes.mark_area_lights(sc)
    far, sc.lights = sc.lights, []
    for k, light in enumerate(far):  # two far lights, one near one, two far lights, ...
        sc.lights.append(light)
        if k % 2:
            pos = tuple(float(x) for x in rng.uniform((-4, 1.5, -4), (4, 2.8, 4)))
            sc.lights.append(Light(type=POINT if k % 4 == 1 else SPOT, position=pos, direction=(0.0, -1.0, 0.0),
                                   intensity=2e-4, cos_inner_cone=0.9, cos_outer_cone=0.2))
    return sc


@pytest.mark.parametrize("areas,spp,nls", [(2, 32, 1), (4, 32, 2), (8, 64, 1), (8, 40, 1), (3, 33, 1)])
def test_lanes_disagree_on_pairs(gpu_ctx, areas, spp, nls):
    out = []
    for pad in (0, 40):
        sc = far_lit_room(areas)
        sc.lights += [Light(type=POINT, position=(0.0, 2.0, 0.0), intensity=0.0) for _ in range(pad)]
        rc = api.RasterConfig(48, 48, 1)
        ds = api.DeviceScene(gpu_ctx, sc)
        pts = api.RasterizeScene(ds, rc, ctx=gpu_ctx)
        out.append(api.BakeSHLightMap(ds, pts, rc, api.BakeConfig(samples=spp, bounces=1, seed=8, num_light_samples=nls),
                                      ctx=gpu_ctx).sh_texture)
    assert np.abs(out[0]).max() > 0 and out[0].tobytes() == out[1].tobytes()
