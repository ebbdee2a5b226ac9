"""The batch autotuner's file across builds: a choice that another build's
kernels were timed for is searched for again, not taken over."""
import pytest

from sh_baker_b200 import api, scenes
from sh_baker_b200 import build as B


def test_kernel_id_follows_sources_and_flags(tmp_path, monkeypatch):
    one = B.kernel_id()
    assert one == B.kernel_id() and " " not in one and "|" not in one
    assert len({one, B.kernel_id(["SHB_REFILL_MIN=8"]), B.kernel_id(file_flags={"shade.cu": ["-fmad=true"]})}) == 3
    for f in B.KERNELS:
        (tmp_path / f).write_bytes((B.CSRC / f).read_bytes())
    monkeypatch.setattr(B, "CSRC", tmp_path)
    assert B.kernel_id() == one
    for f in B.KERNELS:
        (tmp_path / f).write_text((tmp_path / f).read_text() + "// changed\n")
        changed = B.kernel_id()
        assert changed != one
        one = changed


@pytest.mark.gpu
@pytest.mark.parametrize("build", ["v2", "k000000000000"])
def test_choices_of_other_builds_are_not_taken(gpu_ctx, tmp_path, build):
    ds = api.DeviceScene(gpu_ctx, scenes.procedural_room(seed=3, n_boxes=6, res=32))
    rc = api.RasterConfig(32, 32, 1)
    bake = api.BatchBake(ds, api.rasterize_to_device(ds, rc), rc, api.BakeConfig(samples=16, bounces=1, seed=1))
    cache = tmp_path / "tune.txt"
    api.bake_batch(gpu_ctx, [bake], autotune=True, tune_cache=str(cache))
    key = cache.read_text().split()[0].split("|")
    assert len(key) == 3 and key[1] == B.kernel_id()
    old = f"{key[0]}|{build}|{key[2]} 32 1 1 0 0.5\n"  # 32 paths a wave: hundreds of waves
    cache.write_text(old)
    _, st = api.bake_batch(gpu_ctx, [bake], autotune=True, tune_cache=str(cache))
    lines = cache.read_text().splitlines()
    assert st.waves == 1 and lines[0] + "\n" == old and len(lines) == 2 and lines[1].split("|")[1] == key[1]
    _, st = api.bake_batch(gpu_ctx, [bake], autotune=True, tune_cache=str(cache))
    assert st.waves == 1 and cache.read_text().splitlines() == lines
