"""pack_scene takes and refuses what setting the descriptor's fields one by
one takes and refuses: a geometry without vertices is a TypeError, and a
material id is the low 32 bits of whatever integer it is given as (an
unsigned -1 among them)."""
import numpy as np
import pytest

from sh_baker_b200.scene import Geometry, Material, Scene, pack_scene

TRI = dict(vertices=np.eye(3, dtype=np.float32), indices=np.arange(3, dtype=np.uint32))


def test_missing_vertices_are_refused():
    for indices in (np.zeros(0, np.uint32), np.arange(3, dtype=np.uint32)):
        with pytest.raises(TypeError):
            pack_scene(Scene([Geometry(vertices=None, indices=indices)], [], []))


@pytest.mark.parametrize("given,packed", [(0, 0), (-1, -1), (np.uint32(0xFFFFFFFF), -1), (2 ** 32 + 3, 3),
                                          (np.int64(7), 7), (2 ** 31, -2 ** 31)])
def test_material_ids_wrap(given, packed):
    desc, keep = pack_scene(Scene([Geometry(**TRI, material_id=given)], [Material()], []))
    assert desc.geometries[0].material_id == packed and keep


def test_forms_of_arrays():
    forms = [TRI["vertices"], np.asfortranarray(TRI["vertices"]), TRI["vertices"].astype(np.float64),
             TRI["vertices"].astype(">f4"), TRI["vertices"].reshape(-1), TRI["vertices"].tolist(),
             np.repeat(TRI["vertices"], 2, axis=1)[:, ::2]]
    for v in forms:
        desc, keep = pack_scene(Scene([Geometry(vertices=v, indices=[[0, 1, 2]], normals=v)], [], []))
        d = desc.geometries[0]
        assert d.vertex_count == 3 and d.index_count == 3 and keep
        assert d.vertices[0:9] == np.eye(3).reshape(-1).tolist() == d.normals[0:9]
        assert d.indices[0:3] == [0, 1, 2] and not d.texture_uvs
        assert list(d.transform) == [1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0]
