"""Which passes end in the launch that traces the last paths: those whose camera
rays all fit it need no wave (one launch, counted as one wave), one path more runs
waves first (four to a graph), and passes that are counted or guided run waves
only.  With this the comparisons of test_gpu_tail.py are known to compare two
routes, on both sides of the 6,144 rays."""
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def waves(w, h, flags=cb.COMPAT_ALL, setup=None, spp=1, **kw):
    it = cb.load_scene(scenes.config1(5, w, h), flags=flags, max_depth=9, **kw)
    if setup:
        setup(it)
    it.render(spp)
    n = it.stats()["waves"]
    it.close()
    return n


@pytest.mark.parametrize("two", [0, cb.TWO_LEVEL])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (6143, 1), (96, 64)])
def test_tail_alone(w, h, two):
    assert waves(w, h, cb.COMPAT_ALL | two) == 1
    assert waves(w, h, cb.DOME_ALIAS | two) == 1


@pytest.mark.parametrize("flags", [cb.COMPAT_ALL, cb.DOME_ALIAS, cb.COMPAT_PDF | cb.DOME_ALIAS])
def test_waves_first(flags):
    n = waves(6145, 1, flags)
    assert n >= 4 and n % 4 == 0
    n = waves(96, 64, flags, spp=2)  # 12,288 paths
    assert n >= 4 and n % 4 == 0


def test_counted_and_guided_passes():
    for n in (waves(96, 64, cb.COMPAT_ALL | cb.TRACE_STATS), waves(96, 64, cb.COMPAT_ALL | cb.PROFILE_STAGES),
              waves(96, 64, cb.DOME_ALIAS, lambda it: it.setGuiding(cb.GuideConfig(train_spp=0, log2_table=10)))):
        assert n >= 8 and n % 4 == 0


def test_direct_lighting():
    it = cb.load_scene(scenes.config1(5, 96, 64), cb.IntegratorType.WavefrontDirectLighting)
    it.render(1)
    assert it.stats()["waves"] == 4
    it.close()
