"""Mesh uploads gather arrays below 64 KB in 1 MB blocks: array sizes below, at and
above the limit (5,461 vertices are 65,532 bytes of positions, 5,462 65,544; 8,192
of uvs are 65,536), more small arrays than one block holds, meshes without normals
or uvs between others.  Triangles equal the host's to the last bit; normals and
tangents equal those that an edit writes without gathering (the films' paths are
equal: 8 additions per pixel in any order, 8 roundings of 2^-24)."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def mesh(nv, nt, normals, uvs, rng):
    unit = lambda v: (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    c = rng.uniform([-8, 0.2, -4], [8, 4, 8])
    idx = rng.integers(0, nv, (nt, 3)).astype(np.uint32)
    idx[0] = [0, nv // 2, nv - 1]
    return scenes.Mesh((c + rng.normal(scale=0.8, size=(nv, 3))).astype(np.float32),
                       unit(rng.normal(size=(nv, 3)) + [0, 2, 0]) if normals else None, unit(rng.normal(size=(nv, 3))),
                       rng.random((nv, 2)).astype(np.float32) if uvs else None, idx)


@pytest.mark.parametrize("sizes", [[(3, 1)], [(5461, 5), (5462, 5), (3, 1), (8192, 5461), (8191, 5462), (4, 2)],
                                   [(3, 1)] * 500, [(5000, 3)] * 30 + [(30000, 20)] + [(700, 4000)] * 30])
def test_uploaded_arrays(sizes):
    rng = np.random.default_rng(len(sizes))
    meshes = [mesh(nv, nt, i % 3 != 1, i % 2 == 0, rng) for i, (nv, nt) in enumerate(sizes)]
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 60.0, 48, 48)
    s = scenes.Scene(48, 48, meshes, [(i, 0, scenes.IDENTITY) for i in range(len(meshes))],
                     [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.5, 0.5, 0.5))], [scenes.directional()], cam)
    it = cb.load_scene(s, flags=0)
    t = it.bvh()[1]
    got = np.empty((len(t), 3, 3), np.float32)
    got[t[:, 3].view(np.uint32)] = t.reshape(-1, 3, 4)[:, :, :3]
    np.testing.assert_array_equal(got, np.concatenate([m.positions[m.indices.astype(np.int64)] for m in meshes]))
    it.render(8)
    a = it.readbackFramebuffer().copy()
    for i in range(0, len(meshes), max(1, len(meshes) // 40)):
        it.updateVertices(i, meshes[i].positions, meshes[i].normals, meshes[i].tangents, bvh="refit")
    it.render(8)
    b = it.readbackFramebuffer()
    assert len(sizes) == 1 or a[..., :3].max() > 0  # one triangle may be out of view
    np.testing.assert_allclose(a, b, rtol=8 * 2.0 ** -24 * 2, atol=1e-7)
    it.close()
