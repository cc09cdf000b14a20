"""Ray query kernels at the sizes where they can go wrong: one ray, around a
warp, more rays than one upload holds (2^21).  Every ray is one of 1,000 base
rays, whose results the other tests check against the oracle, so each result
must equal its base ray's exactly; a ray is occluded where it has a hit."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, cb.TWO_LEVEL])
def scene(request):
    it = cb.load_scene(scenes.config1(3, 16, 16), flags=cb.COMPAT_ALL | request.param)
    rng = np.random.default_rng(8)
    o = rng.uniform([-5, 0.2, -5], [5, 3, 5], (1000, 3))
    d = rng.normal(size=(1000, 3))
    rays = np.concatenate([o, np.full((1000, 1), 1e-3), d, np.full((1000, 1), 20.0)], 1).astype(np.float32)
    yield it, rays, it.traceRays(rays)
    it.close()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4099, (1 << 21) - 1, (1 << 21) + 5])
def test_query_sizes(scene, n):
    it, base, want = scene
    at = np.arange(n) * 7 % 1000
    rays = base[at]
    got = it.traceRays(rays)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w[at])
    occ = it.occludedRays(rays)
    np.testing.assert_array_equal(occ, (want[1][at] != 0xFFFFFFFF).astype(np.uint8))


@pytest.mark.parametrize("k", [-60, -7, 40, 122, 124])
def test_scaled_directions(scene, k):
    """A direction scaled by 2^k gives the same hits with distances scaled by
    2^-k: the box tests' reciprocals, the approximation and (components above
    1e37: 2^124) the quotient, lose none.  Flattened scenes exactly; a two-level
    scene maps the ray first, to the same bits up to a power of two."""
    it, base, _ = scene
    rays = base.copy()
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7], axis=1, keepdims=True)
    rays[::7, 5] = 0.0  # components below the box tests' smallest stay harmless
    rays[:, 3], rays[:, 7] = 0.0, np.float32(3e38)
    t0, p0, a0, b0 = it.traceRays(rays)
    rays[:, 4:7] *= np.float32(2.0) ** np.float32(k)
    t, p, a, b = it.traceRays(rays)
    np.testing.assert_array_equal(p, p0)
    hit = p0 != 0xFFFFFFFF
    assert hit.sum() > 100
    if k <= 40:  # beyond, the triangle test's products (about 2^-k times an area) leave FP32's normal range
        np.testing.assert_array_equal(np.ldexp(t[hit].astype(np.float64), k), t0[hit].astype(np.float64))
    np.testing.assert_array_equal(a, a0)
    np.testing.assert_array_equal(b, b0)
