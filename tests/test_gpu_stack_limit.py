"""Ray queries and renders report a traversal that ran out of stack instead of
counting its rays as misses: with the stacks limited to one entry each call ends in
an error (the kernels check every push), and without the limit the results are
what they were."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import _native as N
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
def test_overflow_is_reported(two):
    it = cb.load_scene(scenes.config1(3, 32, 32), flags=cb.COMPAT_ALL | two)
    rng = np.random.default_rng(8)
    rays = np.concatenate([rng.uniform([-5, 0.2, -5], [5, 3, 5], (1000, 3)), np.full((1000, 1), 1e-3),
                           rng.normal(size=(1000, 3)), np.full((1000, 1), 20.0)], 1).astype(np.float32)
    calls = [it.traceRays, it.occludedRays, it.traceStats, lambda r: it.render(1)]
    want = [c(rays) for c in calls]
    N.call("cl_unit_limit_stack", it._h, 1)
    for c in calls:
        with pytest.raises(cb.ClError, match="stack overflow") as e:
            c(rays)
        assert e.value.status == N.CL_ERR_STATE
    N.call("cl_unit_limit_stack", it._h, 0xFFFFFFFF)
    for c, w in zip(calls[:3], want):
        for a, b in zip(c(rays), w):
            np.testing.assert_array_equal(a, b)
    it.render(1)
    it.close()
