"""kPathTail, the launch that traces the last paths of a pass to their end,
against the wave kernels alone (CL_TRACE_STATS passes never take it): the same
paths, so equal ray counts and FP64 film sums that differ by the order of the
additions only (at most a few hundred additions per pixel: 1e-12 relative would
do; 1e-9 is asserted).  Sizes: one path, fewer paths than warps, one path below,
at and above the queue length that the tail takes at once, and passes that reach
it after several waves, with and without path regeneration."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu
TAIL = 6144


def render(s, spp, flags, **kw):
    it = cb.load_scene(s, flags=flags | cb.FILM_FP64, **kw)
    it.render(spp)
    s1, s2 = it.readbackFilmStats()
    st = it.stats()
    it.close()
    return s1, s2, st


@pytest.mark.parametrize("w,h,spp,slots", [(1, 1, 1, 0), (7, 5, 1, 0), (33, 31, 3, 0), (TAIL - 1, 1, 1, 0), (96, 64, 1, 0),
                                           (TAIL + 1, 1, 1, 0), (256, 200, 2, 0), (300, 200, 2, 30011)])
@pytest.mark.parametrize("flags", [cb.COMPAT_ALL, cb.DOME_ALIAS, cb.COMPAT_PDF | cb.DOME_ALIAS])
def test_tail_equals_waves(w, h, spp, slots, flags):
    s = scenes.config1(5, w, h)
    a1, a2, sa = render(s, spp, flags, path_slots=slots, max_depth=9)
    b1, b2, sb = render(s, spp, flags | cb.TRACE_STATS, path_slots=slots, max_depth=9)
    assert sa["last_rays_closest"] == sb["last_rays_closest"] and sa["last_rays_shadow"] == sb["last_rays_shadow"]
    np.testing.assert_allclose(a1, b1, rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(a2, b2, rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
def test_tail_equals_waves_instances(two):
    s = scenes.config1(6, 90, 80)
    rng = np.random.default_rng(3)
    for i in range(1, len(s.instances)):
        mesh, mat, _ = s.instances[i]
        q, _r = np.linalg.qr(rng.normal(size=(3, 3)))
        m = np.concatenate([q * rng.uniform(0.6, 1.4), rng.uniform(-1, 1, (3, 1))], 1)
        s.instances[i] = (mesh, mat, tuple(float(x) for x in m.reshape(-1)))
    a1, _, sa = render(s, 2, cb.DOME_ALIAS | two, max_depth=16)
    b1, _, sb = render(s, 2, cb.DOME_ALIAS | two | cb.TRACE_STATS, max_depth=16)
    assert sa["last_rays_closest"] == sb["last_rays_closest"] and sa["last_rays_shadow"] == sb["last_rays_shadow"]
    np.testing.assert_allclose(a1, b1, rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("slots", [0, 4099])
def test_tail_radiance_cache(slots):
    """Training paths end in the tail; every other path has had its cache query
    by then.  Paths do not depend on the predictions, so the counts are equal;
    the predictions after a training step may differ in the last BF16 bit (the
    gradient's order of addition), 2^-8 of the cache's share of the film."""
    s = scenes.config1(7, 128, 96, glass_frac=0.6, glass_alpha=(0.01, 0.1))
    got = []
    for extra in (0, cb.TRACE_STATS):
        it = cb.load_scene(s, flags=cb.DOME_ALIAS | cb.FILM_FP64 | extra, max_depth=16, path_slots=slots)
        it.setRadianceCache(cb.RadianceCacheConfig(train_spp=2))
        it.render(3)
        got.append((it.readbackFilmStats()[0], it.stats(), it.cacheStats()))
        it.close()
    (a, sa, ca), (b, sb, cc) = got
    assert sa["last_rays_closest"] == sb["last_rays_closest"] and sa["last_rays_shadow"] == sb["last_rays_shadow"]
    assert ca["inferred"] == cc["inferred"] and ca["records_last"] == cc["records_last"]
    assert np.linalg.norm(a - b) <= 2.0 ** -8 * np.linalg.norm(b)
