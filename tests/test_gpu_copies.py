"""A vertex edit writes all copies of the mesh in one launch: after it every
triangle of the scene equals that of a scene opened with the new vertices, to the
last bit (the same kernel arithmetic).  One copy, copies whose vertices end before,
at and after a block of 256, thousands, and copies interleaved with other meshes'."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def scene(copies, mesh, rng):
    tri = scenes.Mesh(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0.5]], np.float32), None,
                      np.tile(np.float32([1, 0, 0]), (3, 1)), None, np.array([[0, 1, 2]], np.uint32))
    meshes = [scenes.quad_mesh(20.0), tri, scenes.sphere_mesh(0, (0, 0, 0), 0.5)]
    inst = [(0, 0, scenes.IDENTITY)]
    for i in range(copies):
        m = np.concatenate([np.linalg.qr(rng.normal(size=(3, 3)))[0] * rng.uniform(0.5, 2.0), rng.uniform(-9, 9, (3, 1))], 1)
        inst.append((mesh, 0, tuple(float(x) for x in m.reshape(-1))))
        if i % 3 == 0:
            inst.append((3 - mesh, 0, tuple(float(x) for x in m.reshape(-1))))
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 45.0, 16, 16)
    return scenes.Scene(16, 16, meshes, inst, [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.5, 0.5, 0.5))],
                        [scenes.directional()], cam)


def triangles(it):
    t = it.bvh()[1]
    out = np.empty((len(t), 3, 3), np.float32)
    out[t[:, 3].view(np.uint32)] = t.reshape(-1, 3, 4)[:, :, :3]
    return out


@pytest.mark.parametrize("mesh,copies", [(1, 1), (1, 2), (1, 85), (1, 86), (1, 171), (2, 1), (2, 21), (2, 22), (2, 4000)])
def test_edit_of_all_copies(mesh, copies):
    rng = np.random.default_rng(copies)
    s = scene(copies, mesh, rng)
    it = cb.load_scene(s)
    m = s.meshes[mesh]
    m.positions = (m.positions + rng.normal(scale=0.05, size=m.positions.shape)).astype(np.float32)
    it.updateVertices(mesh, m.positions, bvh="refit")
    got = triangles(it)
    it.close()
    fresh = cb.load_scene(s)
    np.testing.assert_array_equal(got, triangles(fresh))
    fresh.close()


def test_edit_of_a_mesh_without_copies():
    s = scene(5, 1, np.random.default_rng(0))
    s.instances = [i for i in s.instances if i[0] != 2]
    it = cb.load_scene(s)
    before = triangles(it)
    it.updateVertices(2, s.meshes[2].positions * np.float32(2.0), bvh="refit")
    np.testing.assert_array_equal(triangles(it), before)
    it.close()
