"""Network entry points over calls of changing size: the staging buffers are
kept between calls and the records are packed on the device, so each result must
equal that of a network that makes this call alone (forward, sample and pdf to
the last bit; gradients by their order of addition: 1e-5 of the largest)."""
import numpy as np
import pytest

import colvillea_b200 as cb

pytestmark = pytest.mark.gpu
CFG = dict(log2_table=10, batch=512)


def rows(n, rng, k):
    r = rng.normal(size=(n, k)).astype(np.float32)
    r[:, :3] = rng.random((n, 3))
    for a in (3, 6, 9):
        if a + 3 <= k and not (k == 12 and a == 9):
            r[:, a:a + 3] /= np.linalg.norm(r[:, a:a + 3], axis=1, keepdims=True)
    r[:, 9 if k == 12 else 12:] = np.abs(r[:, 9 if k == 12 else 12:]) + np.float32(0.1)
    return r


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
def test_guide_calls(n):
    rng = np.random.default_rng(n)
    rec, big = rows(n, rng, 14), rows(700, rng, 14)
    u3 = rng.random((n, 3)).astype(np.float32)
    used, fresh = cb.Guide.create(cb.GuideConfig(**CFG)), [cb.Guide.create(cb.GuideConfig(**CFG)) for _ in range(4)]
    used.gradient(big); used.forward(big[:, :9]); used.sample(big[:3, :9], rng.random((3, 3)))
    in9 = np.ascontiguousarray(rec[:, :9])
    np.testing.assert_array_equal(used.forward(in9), fresh[0].forward(in9))
    for a, b in zip(used.sample(in9, u3), fresh[1].sample(in9, u3)):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(used.pdf(in9, rec[:, 9:12]), fresh[2].pdf(in9, rec[:, 9:12]))
    (la, ga), (lb, gb) = used.gradient(rec), fresh[3].gradient(rec)
    assert abs(la - lb) <= 1e-5 * abs(lb) and np.abs(ga - gb).max() <= 1e-5 * np.abs(gb).max()
    for g in [used, *fresh]:
        g.close()


@pytest.mark.parametrize("n", [1, 200, 513])
def test_cache_calls(n):
    rng = np.random.default_rng(n)
    rec, big = rows(n, rng, 12), rows(600, rng, 12)
    net = cb.RadianceCacheConfig(network=CFG).network
    used, fresh = cb.Cache.create(net), cb.Cache.create(net)
    used.gradient(big); used.forward(big[:, :9])
    np.testing.assert_array_equal(used.forward(rec[:, :9]), fresh.forward(rec[:, :9]))
    (la, ga), (lb, gb) = used.gradient(rec), fresh.gradient(rec)
    assert abs(la - lb) <= 1e-5 * abs(lb) and np.abs(ga - gb).max() <= 1e-5 * np.abs(gb).max()
    used.close(); fresh.close()
