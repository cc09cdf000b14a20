"""Device allocations that fail, injected on the host (from the given one on, so
that what a call repeats with more room fails too): the call reports CL_ERR_OOM,
what follows uses nothing of what it replaced, and the same call succeeds
afterwards with the results that it has always had."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import _native as N
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def failing(after, call):
    N.call("cl_unit_fail_allocations", after, 1000)
    try:
        with pytest.raises(cb.ClError) as e:
            call()
        assert e.value.status == N.CL_ERR_OOM
    finally:
        N.call("cl_unit_fail_allocations", 0, 0)


def test_dome_build():
    """A larger dome that does not fit: no emitters are left (a dark film), neither
    the old dome's tables nor the captured graph that pointed at them."""
    s = scenes.config1(4, 48, 48)
    it = cb.load_scene(s)
    it.render(1)
    want = it.readbackFramebuffer().copy()
    big = scenes.Emitter(scenes.EMIT_DOME, texels=np.ones((256, 512, 4), np.float32))
    failing(0, lambda: it.buildEmitters([big]))
    it.resetIterationIndex(); it.render(1)
    assert (it.readbackFramebuffer()[..., :3] == 0).all()
    it.buildEmitters(s.emitters)
    it.resetIterationIndex(); it.render(1)
    np.testing.assert_array_equal(it.readbackFramebuffer(), want)  # one path per pixel
    it.close()


@pytest.mark.parametrize("mode", ["plain", "guide", "cache"])
def test_first_render(mode):
    """Each allocation of a first render fails in turn; the render that follows has
    the same paths (and, where no network trains, the same film)."""
    s = scenes.config1(4, 48, 48)

    def make():
        it = cb.load_scene(s, flags=cb.DOME_ALIAS | cb.FILM_FP64, path_slots=4096)
        if mode == "guide":
            it.setGuiding(cb.GuideConfig(train_spp=0, log2_table=10))
        elif mode == "cache":
            it.setRadianceCache(cb.RadianceCacheConfig(train_spp=1, network={"batch": 512, "log2_table": 10}))
        return it

    def result(it):
        it.render(1)
        st = it.stats()
        film = it.readbackFilmStats()[0].copy()
        it.close()
        return (st["last_rays_closest"], st["last_rays_shadow"]), film

    rays, film = result(make())
    after = 0
    while True:
        it = make()
        N.call("cl_unit_fail_allocations", after, 1000)
        try:
            it.render(1)
            done = True
        except cb.ClError as e:
            assert e.status == N.CL_ERR_OOM
            done = False
        N.call("cl_unit_fail_allocations", 0, 0)
        if done:
            it.close()
            break
        got, f = result(it)
        assert got == rays
        if mode != "cache":
            np.testing.assert_allclose(f, film, rtol=1e-9, atol=1e-12)
        assert np.isfinite(f).all()
        after += 1
    assert after == {"plain": 3, "guide": 6, "cache": 8}[mode]  # film, FP64 film, queues, the network's buffers


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
def test_rebuild_after_edit(two):
    """Each allocation of a rebuild fails in turn: the new vertices have no tree then,
    so a render is refused until the instances are built again."""
    s = scenes.config1(4, 32, 32)
    m = s.meshes[1]
    moved = (m.positions + np.float32(0.1)).astype(np.float32)
    fresh = scenes.config1(4, 32, 32)
    fresh.meshes[1].positions = moved
    it = cb.load_scene(fresh, flags=cb.COMPAT_ALL | two)
    it.render(1)
    want = it.readbackFramebuffer().copy()
    it.close()
    it = cb.load_scene(s, flags=cb.COMPAT_ALL | two)
    it.render(1)
    for after in range(3):
        failing(after, lambda: it.updateVertices(1, moved, bvh="rebuild"))
        with pytest.raises(cb.ClError) as e:
            it.render(1)
        assert e.value.status == N.CL_ERR_STATE
        it.buildTLAS(s.instances)
        it.resetIterationIndex(); it.render(1)
        np.testing.assert_allclose(it.readbackFramebuffer(), want, rtol=1e-6)
    it.updateVertices(1, m.positions); it.updateVertices(1, moved, bvh="rebuild")
    it.render(1)
    np.testing.assert_allclose(it.readbackFramebuffer(), want, rtol=1e-6)
    it.close()


def test_auto_keeps_a_refitted_tree():
    """The rebuild that an automatic update adds finds no memory: the error is
    reported, and the refitted tree serves the new vertices."""
    def scene():
        s = scenes.config1(4, 32, 32)
        s.meshes[1] = scenes.sphere_mesh(4, (0, 1, 0), 1.0)
        return s

    p = scene().meshes[1].positions
    p = p[np.random.default_rng(1).permutation(len(p))] * np.float32(4.0)
    ref = cb.load_scene(scene())
    ref.updateVertices(1, p, bvh="auto")
    assert ref.stats()["bvh_rebuilds"] == 1
    it = cb.load_scene(scene())
    failing(0, lambda: it.updateVertices(1, p, bvh="auto"))
    assert it.stats()["bvh_refits"] >= 1 and it.stats()["bvh_rebuilds"] == 0
    rng = np.random.default_rng(2)
    rays = np.concatenate([rng.uniform(-5, 5, (2000, 3)), np.full((2000, 1), 1e-3), rng.normal(size=(2000, 3)),
                           np.full((2000, 1), 1e3)], 1).astype(np.float32)
    for a, b in zip(it.traceRays(rays), ref.traceRays(rays)):
        np.testing.assert_array_equal(a, b)
    it.close(); ref.close()
