"""Rays along an axis, whose zero components may be negative: a directional
light of (0, -1, 0) sends its shadow rays along (-0, 1, -0).  The traversal
takes a component's sign for its reciprocal and for its order of planes, and
both zeros must give the same walk.  Compared with the oracle's closest hits
(the triangle test rounds alike in both, so a ray that hits the same triangle
has the same distance; up to 5 rays in 10,000 may graze an edge) and bakes
(the bounds of the suite's other oracle bakes)."""
import itertools

import numpy as np
import pytest

from oracle import pyoracle as O
from sh_baker_b200 import api, scenes
from sh_baker_b200.scene import DIRECTIONAL, Light

pytestmark = pytest.mark.gpu

ZERO_DIRS = [d for d in itertools.product((0.0, -0.0, 0.7, -0.7), repeat=3) if 0.0 in d and any(d)]


@pytest.mark.parametrize("n_boxes", [0, 40])
def test_zero_components(gpu_ctx, n_boxes):
    sc = scenes.procedural_room(seed=9, n_boxes=n_boxes, res=64)
    rng = np.random.default_rng(3)
    n = 300 * len(ZERO_DIRS)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform((-4.9, 0.1, -4.9), (4.9, 2.9, 4.9), (n, 3))
    rays[:, 3:6] = np.tile(np.float32(ZERO_DIRS), (300, 1))
    rays[:, 6], rays[:, 7] = 0.001, np.inf
    got = api.FindOcclusion(sc, rays, ctx=gpu_ctx)
    want = O.OracleScene(sc).find_occlusion(rays)
    assert (want["hit"] == 1).mean() > 0.99  # a closed room
    same = (got["hit"] == want["hit"]) & (got["prim_id"] == want["prim_id"])
    assert (~same).sum() <= 5e-4 * n
    assert np.array_equal(got["t"][same], want["t"][same])


def test_both_zeros_are_one_ray(gpu_ctx):
    # also from points on the walls and on box faces, along them
    sc = scenes.procedural_room(seed=9, n_boxes=40, res=64)
    rng = np.random.default_rng(5)
    verts = np.concatenate([g.vertices for g in sc.geometries])
    rays = np.empty((4096, 8), np.float32)
    rays[:, 0:3] = verts[rng.integers(0, len(verts), 4096)] * rng.choice([1.0, 0.5], (4096, 3))
    rays[:, 3:6] = rng.choice([0.0, 0.7, -0.7], (4096, 3))
    rays[np.all(rays[:, 3:6] == 0.0, 1), 4] = 1.0
    rays[:, 6], rays[:, 7] = 0.001, np.inf
    hits = []
    for zero in (0.0, -0.0):
        r = rays.copy()
        r[:, 3:6][r[:, 3:6] == 0.0] = zero
        hits.append(api.FindOcclusion(sc, r, ctx=gpu_ctx))
    assert (hits[0]["hit"] == 1).any()
    for name in ("hit", "t", "prim_id", "uv"):
        assert hits[0][name].tobytes() == hits[1][name].tobytes(), name


@pytest.mark.parametrize("direction", [(0.0, -1.0, 0.0), (-0.0, -1.0, 0.0), (-0.6, -0.8, 0.0), (0.0, -0.8, 0.6)])
def test_axis_aligned_sun(gpu_ctx, direction):
    # a furnished room without its ceiling: sunlit floor, shadows of the boxes
    sc = scenes.procedural_room(seed=6, n_boxes=30, res=48, n_point_lights=0)
    for g in sc.geometries:
        tri = np.asarray(g.indices).reshape(-1, 3)
        up = np.asarray(g.vertices)[:, 1][tri].min(1) > 2.99
        g.indices = np.ascontiguousarray(tri[~up].reshape(-1))
    sc.lights = [Light(type=DIRECTIONAL, direction=direction, intensity=3.0)]
    osc = O.OracleScene(sc)
    pts = osc.rasterize(96, 96, 1)
    ref = osc.bake(pts, 96, 96, 1, samples=32, bounces=2, seed=13)
    got = api.BakeSHLightMap(sc, pts, api.RasterConfig(96, 96, 1), api.BakeConfig(samples=32, bounces=2, seed=13),
                             ctx=gpu_ctx)
    # (where the light grazes the surface itself, the shadow ray runs in the
    # wall's plane, and whether it meets an edge there is anyone's guess)
    valid = ((pts["material_id"] >= 0) & (np.abs(pts["normal"] @ np.float32(direction)) > 1e-6)).reshape(96, 96)
    g, r = got.sh_texture[valid].reshape(-1, 27), ref["sh"][valid].reshape(-1, 27)
    assert 0.1 < (np.abs(r).max(1) > 0.5).mean() < 0.97  # lit and shadowed texels
    close = np.isclose(g, r, rtol=1e-3, atol=1e-5).all(axis=1)
    assert close.mean() >= 0.97, close.mean()
    assert np.linalg.norm(g - r) / np.linalg.norm(r) < 2e-2
