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
