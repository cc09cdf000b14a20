"""Flattening, mesh uploads and instance boxes on the device against the host
scene description: scenes.Scene.flatten() holds the world-space arrays (double
arithmetic, rounded once, as the kernels), so the triangles of the built tree
must equal it to the last bit or, where numpy's matrix product adds in another
order, within 1 ulp of the largest term; odd vertex counts, meshes without
normals or uvs, one-triangle meshes and many copies of one mesh."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def scene(copies, rng):
    tri = scenes.Mesh(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0.5]], np.float32), None,
                      np.tile(np.float32([1, 0, 0]), (3, 1)), None, np.array([[0, 1, 2]], np.uint32))
    meshes = [scenes.quad_mesh(20.0), tri, scenes.sphere_mesh(1, (0, 0, 0), 0.5), scenes.torus_mesh(17, 13, (0, 0, 0), 0.6, 0.2)]
    inst = [(0, 0, scenes.IDENTITY)]
    for i in range(copies):
        m = np.concatenate([np.linalg.qr(rng.normal(size=(3, 3)))[0] * rng.uniform(0.5, 2.0), rng.uniform(-4, 4, (3, 1))], 1)
        inst.append((1 + i % 3, i % 2, tuple(float(x) for x in m.astype(np.float32).reshape(-1))))
    mats = [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.5, 0.5, 0.5)),
            scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.8, 0.2, 0.2))]
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 45.0, 32, 32)
    return scenes.Scene(32, 32, meshes, inst, mats, [scenes.directional()], cam)


def triangles(s):
    out = []
    for mesh_id, _, xf in s.instances:
        m = s.meshes[mesh_id]
        M = np.asarray(xf, np.float32).astype(np.float64).reshape(3, 4)
        p = m.positions.astype(np.float64)
        w = ((p[:, :1] * M[:, 0] + p[:, 1:2] * M[:, 1]) + p[:, 2:] * M[:, 2] + M[:, 3]).astype(np.float32)
        out.append(w[m.indices.astype(np.int64)])
    return np.concatenate(out)


@pytest.mark.parametrize("copies", [1, 2, 64, 1000])
def test_flattened_triangles(copies):
    s = scene(copies, np.random.default_rng(copies))
    it = cb.load_scene(s)
    _, t = it.bvh()
    it.close()
    got = np.empty((len(t), 3, 3), np.float32)
    ids = t[:, 3].view(np.uint32)
    got[ids] = t.reshape(-1, 3, 4)[:, :, :3]
    np.testing.assert_array_equal(got, triangles(s))


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
@pytest.mark.parametrize("mesh", [1, 2, 3])
def test_edit_equals_fresh_scene(two, mesh):
    """New vertices (and normals for a mesh that had none): closest hits and the
    film equal those of a scene opened with them (hits exactly; film by the
    order of its additions)."""
    rng = np.random.default_rng(mesh)
    s = scene(24, rng)
    it = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    m = s.meshes[mesh]
    m.positions = (m.positions * np.float32(1.25) + rng.normal(scale=0.02, size=m.positions.shape)).astype(np.float32)
    m.normals = np.tile(np.float32([0, 1, 0]), (len(m.positions), 1)) if m.normals is None else m.normals
    it.updateVertices(mesh, m.positions, m.normals)
    fresh = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    o = rng.uniform(-5, 5, (5000, 3))
    rays = np.concatenate([o, np.full((5000, 1), 1e-3), rng.normal(size=(5000, 3)), np.full((5000, 1), 1e3)], 1)
    for a, b in zip(it.traceRays(rays.astype(np.float32)), fresh.traceRays(rays.astype(np.float32))):
        np.testing.assert_array_equal(a, b)
    it.render(2); fresh.render(2)
    np.testing.assert_allclose(it.readbackFramebuffer(), fresh.readbackFramebuffer(), rtol=1e-5, atol=1e-6)
    it.close(); fresh.close()


def test_refusals():
    s = scene(3, np.random.default_rng(0))
    it = cb.load_scene(s)
    before = it.bvh()[1]
    bad = scenes.Mesh(s.meshes[1].positions, None, s.meshes[1].tangents, None, np.array([[0, 1, 3]], np.uint32))
    with pytest.raises(cb.ClError, match="mesh 1: vertex index out of range"):
        it.buildBLAS([s.meshes[0], bad, bad])
    p = s.meshes[2].positions.copy()
    p[5, 1] = np.inf
    p[9, 0] = np.nan
    with pytest.raises(cb.ClError, match="vertex 5: position is not finite"):
        it.updateVertices(2, p)
    it.updateVertices(2, s.meshes[2].positions, bvh="refit")  # the refused edits changed nothing
    np.testing.assert_array_equal(it.bvh()[1], before)
    with pytest.raises(cb.ClError, match="instance 1: singular transform"):
        it.buildTLAS([(0, 0, scenes.IDENTITY), (2, 0, (0.0,) * 12)])
    it.render(1)
    it.close()
