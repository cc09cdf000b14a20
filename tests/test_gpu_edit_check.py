"""Vertex edits on both sides of the size from which the finiteness check runs on
the device instead of the host (32,768 floats): a refused edit names the first bad
vertex and changes nothing, an accepted one equals a scene opened with the new
vertices, normals and tangents."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
@pytest.mark.parametrize("nv", [3, 10922, 10923])
def test_edit_check(nv, two):
    rng = np.random.default_rng(nv)
    pos = np.tile(np.float32([0, 0.5, 0]), (nv, 1))
    pos[[0, nv // 2, nv - 1]] = [[-4, 0.5, -4], [4, 0.5, -4], [0, 3, 6]]
    mesh = scenes.Mesh(pos, None, np.tile(np.float32([1, 0, 0]), (nv, 1)), None,
                       np.array([[0, nv // 2, nv - 1]], np.uint32))
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 45.0, 32, 32)
    s = scenes.Scene(32, 32, [scenes.quad_mesh(20.0), mesh], [(0, 0, scenes.IDENTITY), (1, 0, scenes.IDENTITY)],
                     [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.5, 0.5, 0.5))], [scenes.directional()], cam)
    it = cb.load_scene(s, flags=two)
    rays = np.concatenate([rng.uniform(-4, 4, (500, 3)), np.full((500, 1), 1e-3), rng.normal(size=(500, 3)),
                           np.full((500, 1), 1e3)], 1).astype(np.float32)
    before = it.traceRays(rays)
    for bad in (nv - 1, 0):
        p = pos + np.float32(0.25)
        p[bad:, 1] = np.nan if bad else -np.inf
        with pytest.raises(cb.ClError, match=f"vertex {bad}: position is not finite"):
            it.updateVertices(1, p)
        for a, b in zip(it.traceRays(rays), before):
            np.testing.assert_array_equal(a, b)
    mesh.positions = pos + np.float32(0.25)
    mesh.normals = np.tile(np.float32([0, 0.6, -0.8]), (nv, 1))
    mesh.tangents = np.tile(np.float32([0, 0.8, 0.6]), (nv, 1))
    it.updateVertices(1, mesh.positions, mesh.normals, mesh.tangents)
    fresh = cb.load_scene(s, flags=two)
    for a, b in zip(it.traceRays(rays), fresh.traceRays(rays)):
        np.testing.assert_array_equal(a, b)
    it.render(4); fresh.render(4)  # equal paths: the order of a pixel's additions, 4 of them
    np.testing.assert_allclose(it.readbackFramebuffer(), fresh.readbackFramebuffer(), rtol=4e-7, atol=1e-7)
    it.close(); fresh.close()
