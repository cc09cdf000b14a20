"""Meshes without room on the device: the pool goes to host memory when it is
uploaded, or when a later call finds no room beside it (allocations fail on the
host, once each); builds, edits and refusals are those of a pool on the device, to
the last bit of the hits.  And more triangles than a 31-bit count holds, most of
them in meshes that no instance uses."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import _native as N
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def fail_once(after, call):
    N.call("cl_unit_fail_allocations", after, 1)
    try:
        return call()
    finally:
        N.call("cl_unit_fail_allocations", 0, 0)


def scene():
    """A quad, 10,242-vertex and 92-vertex meshes; rotated copies."""
    rng = np.random.default_rng(5)
    meshes = [scenes.quad_mesh(20.0), scenes.sphere_mesh(5, (0, 0, 0), 0.6), scenes.torus_mesh(9, 7, (0, 0, 0), 0.6, 0.2)]
    inst = [(0, 0, scenes.IDENTITY)]
    for i in range(10):
        m = np.concatenate([np.linalg.qr(rng.normal(size=(3, 3)))[0], rng.uniform([-4, 0.5, -4], [4, 3, 4])[:, None]], 1)
        inst.append((1 + i % 2, 0, tuple(float(x) for x in m.astype(np.float32).reshape(-1))))
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 45.0, 32, 32)
    return scenes.Scene(32, 32, meshes, inst, [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.5, 0.5, 0.5))],
                        [scenes.directional()], cam)


def edits(s):
    rng = np.random.default_rng(6)
    out = []
    for mesh, normals in ((2, False), (1, True)):
        p = s.meshes[mesh].positions
        out.append((mesh, (p + rng.normal(scale=0.02, size=p.shape)).astype(np.float32),
                    np.tile(np.float32([0, 1, 0]), (len(p), 1)) if normals else None))
    return out


def results(it):
    rng = np.random.default_rng(7)
    rays = np.concatenate([rng.uniform(-5, 5, (3000, 3)), np.full((3000, 1), 1e-3), rng.normal(size=(3000, 3)),
                           np.full((3000, 1), 1e3)], 1).astype(np.float32)
    it.resetIterationIndex(); it.render(1)
    return [*it.traceRays(rays), it.readbackFramebuffer().copy()]


def equal(a, b):
    for x, y in zip(a[:-1], b[:-1]):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_allclose(a[-1], b[-1], rtol=1e-6)


def open_empty(s, two):
    it = cb.Integrator.createIntegrator(cb.IntegratorType.WavefrontPathTracing, s.width, s.height,
                                        cb.RenderConfig(flags=cb.COMPAT_ALL | two))
    it.buildMaterials(s.materials); it.buildEmitters(s.emitters); it.updateCamera(s.camera)
    return it


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
def test_pool_in_host_memory(two):
    s = scene()
    want = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    it = open_empty(s, two)
    bad = scenes.Mesh(s.meshes[2].positions, None, s.meshes[2].tangents, None, s.meshes[2].indices + np.uint32(60))
    with pytest.raises(cb.ClError, match="mesh 1: vertex index out of range"):
        fail_once(0, lambda: it.buildBLAS([s.meshes[0], bad, bad]))
    fail_once(0, lambda: it.buildBLAS(s.meshes))
    it.buildTLAS(s.instances)
    equal(results(it), results(want))
    for mesh, p, n in edits(s):
        q = p.copy()
        q[-1, 2] = np.nan
        with pytest.raises(cb.ClError, match=f"vertex {len(p) - 1}: position is not finite"):
            it.updateVertices(mesh, q)
        for bvh in ("refit", "rebuild"):
            it.updateVertices(mesh, p, n, bvh=bvh); want.updateVertices(mesh, p, n, bvh=bvh)
            equal(results(it), results(want))
    it.buildBLAS(s.meshes); it.buildTLAS(s.instances)  # and back to the device
    fresh = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    equal(results(it), results(fresh))
    for i in (it, want, fresh):
        i.close()


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
def test_calls_that_find_no_room(two):
    """One allocation of each call fails: the meshes move to host memory, and the call
    succeeds at the second go."""
    s = scene()
    want = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    ref = results(want)
    (mesh, p, n), = edits(s)[1:]
    want.updateVertices(mesh, p, n, bvh="rebuild")
    edited = results(want)
    want.close()
    for after in range(4):
        it = open_empty(s, two)
        it.buildBLAS(s.meshes)
        fail_once(after, lambda: it.buildTLAS(s.instances))
        equal(results(it), ref)
        it.updateVertices(mesh, p, n, bvh="rebuild")
        equal(results(it), edited)
        it.close()
        it = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
        it.render(1)
        fail_once(after % 3, lambda: it.updateVertices(mesh, p, n, bvh="rebuild"))
        equal(results(it), edited)
        it.close()
        it = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
        fail_once(after % 2, lambda: it.render(1))
        equal(results(it), ref)
        it.close()


def test_more_triangles_than_31_bits():
    """257 meshes of 2^23 triangles (one shared array of indices) before the scene's own."""
    s = scene()
    want = cb.load_scene(s)
    ref = results(want)
    want.close()
    tri = s.meshes[0]
    big = scenes.Mesh(tri.positions, None, tri.tangents, None, np.zeros((1 << 23, 3), np.uint32))
    it = open_empty(s, 0)
    it.buildBLAS([big] * 257 + s.meshes)
    it.buildTLAS([(m + 257, mat, xf) for m, mat, xf in s.instances])
    equal(results(it), ref)
    it.close()
