"""The box tests' reciprocals (hardware approximation, one Newton step) against the
IEEE quotient 1/x, to which they have to be within one unit in the last place: all
2^23 mantissas of one binade, many of each other binade from the smallest component
that counts (1e-30) to the switch to the quotient (1e37), both signs; and exactly
the quotient beyond, for zero, subnormal and infinite components."""
import numpy as np
import pytest

from colvillea_b200 import _native as N
from gpu_util import P

pytestmark = pytest.mark.gpu


def inverse(x):
    x = np.ascontiguousarray(x, np.float32).reshape(-1, 3)
    out = np.empty_like(x)
    N.call("cl_unit_box_reciprocals", P(x), P(out), len(x))
    return out.reshape(-1)


def ulps(x):
    got, want = inverse(x), np.float32(1.0) / np.asarray(x, np.float32)
    assert (np.signbit(got) == np.signbit(want)).all()
    d = np.abs(got.view(np.int32).astype(np.int64) - want.view(np.int32))
    return d


def test_all_mantissas():
    m = (np.arange(1 << 23, dtype=np.uint32) | (127 << 23)).view(np.float32)
    m = np.append(m, np.float32(2.0))  # a multiple of 3
    for sign in (1, -1):
        d = ulps(np.float32(sign) * m)
        print(f"[ulp] box reciprocals: {np.count_nonzero(d)} of 2^23 mantissas differ, largest {d.max()}")
        assert d.max() <= 1


def test_all_binades():
    rng = np.random.default_rng(0)
    for e in range(28, 250):  # 2^-99 (6e-31, mostly below the smallest) .. 2^122
        x = ((np.uint32(e) << 23) | rng.integers(0, 1 << 23, 3000, dtype=np.uint32)).view(np.float32)
        x = np.where(np.abs(x) < np.float32(1e-30), np.float32(1e-30), x) * np.where(rng.random(3000) < 0.5, 1, -1)
        x = x.astype(np.float32)
        assert ulps(x).max() <= 1


def test_ends_of_the_range():
    tiny = np.float32([0.0, -0.0, 1e-31, -1e-31, 1e-45, -1e-45, 1e-30, -1e-30, 1.0])
    want = np.copysign(np.maximum(np.abs(tiny), np.float32(1e-30)), tiny)
    d = np.abs(inverse(tiny).view(np.int32).astype(np.int64) - (np.float32(1) / want).view(np.int32))
    assert d.max() <= 1
    for big in (1e37, 2e38, np.inf):  # one such component: all three by the quotient
        x = np.float32([big, 0.3, -7.1, 1.7, -big, 3.3, 0.1, -0.9, big])
        np.testing.assert_array_equal(inverse(x), np.float32(1) / x)
