"""Counters and fills that are cleared once instead of before each use: waves
of very different depths one after another (each depth has a counter set of
its own, 30 bounces being the most), and rasters with more triangles than
texels, after a larger one in the same buffers."""
import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from sh_baker_b200 import api, scenes
from sh_baker_b200.scene import Geometry, Material, Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("depths", [(30, 0, 30), (0, 30, 1), (0, 0, 0)])
def test_waves_of_different_depths(gpu_ctx, depths, use_graph):
    bakes, ref = [], []
    for k, d in enumerate(depths):
        ds = api.DeviceScene(gpu_ctx, scenes.procedural_room(seed=40 + k, n_boxes=6, res=16, n_point_lights=2))
        rc = api.RasterConfig(16, 16, 1)
        g = api.rasterize_to_device(ds, rc)
        bakes.append(api.BatchBake(ds, g, rc, api.BakeConfig(samples=70, bounces=d, seed=3 + k)))
        sh = torch.empty(16 * 16 * 27, dtype=torch.float32, device="cuda")
        env = torch.empty(16 * 16, dtype=torch.float32, device="cuda")
        api.bake_plain_device(bakes[-1], sh, env)
        ref.append((sh.cpu().numpy(), env.cpu().numpy()))
    # one bake a wave, then several waves a bake
    for paths in (1 << 16, 1 << 12):
        outs, st = api.bake_batch(gpu_ctx, bakes, use_graph=use_graph, wave_paths=paths, share_paths=-1)
        assert st.error_flags == 0 and st.waves >= 3
        for (sh, env), (rsh, renv) in zip(outs, ref):
            assert sh.cpu().numpy().tobytes() == rsh.tobytes()
            assert env.cpu().numpy().tobytes() == renv.tobytes()


@pytest.mark.parametrize("n", [1, 31, 33, 63, 64, 65, 129])
def test_short_queues(gpu_ctx, n):
    # about one light query per texel and per hit: queues around the entries
    # that a warp fetches at once
    sc = scenes.procedural_room(seed=12, n_boxes=6, res=16, n_point_lights=2)
    rc = api.RasterConfig(n, 1, 1)
    pts = api.RasterizeScene(sc, rc, ctx=gpu_ctx)
    got = api.BakeSHLightMap(sc, pts, rc, api.BakeConfig(samples=1, bounces=1, seed=8), ctx=gpu_ctx)
    ref = O.OracleScene(sc).bake(pts.reshape(-1), n, 1, 1, samples=1, bounces=1, seed=8)
    g, r = got.sh_texture.reshape(n, 27), ref["sh"].reshape(n, 27)
    off = ~np.isclose(g, r, rtol=2e-4, atol=2e-5 * max(1.0, float(np.abs(r).max()))).all(1)
    assert off.sum() <= max(1, n // 50)  # paths that graze an edge
    assert (got.environment_visibility_texture.reshape(-1) != ref["env"].reshape(-1)).sum() <= max(1, n // 50)


@pytest.mark.parametrize("w,h,ss", [(1, 1, 1), (3, 5, 1), (7, 2, 3), (16, 16, 1)])
def test_more_triangles_than_texels(gpu_ctx, w, h, ss):
    rng = np.random.default_rng(w)
    n = 300
    uv = (rng.uniform(0, 1, (n, 1, 2)) + rng.normal(size=(n, 3, 2)) * 0.02).reshape(-1, 2).astype(np.float32)
    nrm = rng.normal(size=(3 * n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    tan = np.hstack([nrm[:, [1, 2, 0]], np.ones((3 * n, 1))])
    sc = Scene([Geometry(vertices=rng.normal(size=(3 * n, 3)).astype(np.float32), normals=nrm.astype(np.float32),
                         tangents=tan.astype(np.float32), lightmap_uvs=uv, texture_uvs=uv,
                         indices=np.arange(3 * n, dtype=np.uint32), material_id=0)], [Material()], [])
    api.RasterizeScene(scenes.unit_quad(), api.RasterConfig(40, 40, 1), ctx=gpu_ctx)
    got = api.RasterizeScene(sc, api.RasterConfig(w, h, ss), ctx=gpu_ctx)
    assert got.tobytes() == O.OracleScene(sc).rasterize(w, h, ss).tobytes()
