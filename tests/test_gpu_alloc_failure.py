"""Device allocations that fail, injected on the host: the call reports CL_ERR_OOM,
what follows uses nothing of what it replaced, and the same call succeeds
afterwards with the results that it has always had."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import _native as N
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def failing(after, call):
    N.call("cl_unit_fail_allocation", after)
    try:
        with pytest.raises(cb.ClError) as e:
            call()
        assert e.value.status == N.CL_ERR_OOM
    finally:
        N.call("cl_unit_fail_allocation", -1)


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
        N.call("cl_unit_fail_allocation", after)
        try:
            it.render(1)
            done = True
        except cb.ClError as e:
            assert e.status == N.CL_ERR_OOM
            done = False
        N.call("cl_unit_fail_allocation", -1)
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
