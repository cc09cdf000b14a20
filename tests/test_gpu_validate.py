"""The validation of built trees checks every word that the traversal follows: a
tree as built passes, and each word put out of step with the others is named."""
import ctypes

import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import _native as N
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tree():
    it = cb.load_scene(scenes.config1(3, 16, 16))
    n20, tris = it.bvh()
    it.close()
    meta = n20.view(np.uint8).reshape(len(n20), 80)[:, 24:32].astype(np.uint32)
    leaf = np.where((n20[:, 3:4] >> (24 + np.arange(8, dtype=np.uint32))) & 1, 0, meta >> 5)
    n24 = np.zeros((len(n20), 24), np.uint32)
    n24[:, :20] = n20
    n24[:, 20] = (leaf << (3 * np.arange(8, dtype=np.uint32))).sum(1)
    for a in range(3):
        n24[:, 21 + a] = ((n20[:, 3] >> (8 * a)) & 255) << 23
    return n24, leaf, np.ascontiguousarray(tris)


def bits(nodes, tris):
    out = ctypes.c_uint32(99)
    nodes, tris = np.ascontiguousarray(nodes, np.uint32), np.ascontiguousarray(tris)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    N.call("cl_unit_validate_bvh", p(nodes), len(nodes), p(tris), len(tris), ctypes.byref(out))
    return out.value


def test_built_tree_is_valid(tree):
    n, leaf, t = tree
    assert bits(n, t) == 0
    assert (leaf.sum(1) > 0).any() and (leaf == 0).any()  # leaves, and inner or empty slots


@pytest.mark.parametrize("word,flip,want", [(21, 1 << 23, 1), (22, 1, 1), (23, 1 << 31, 1), (3, 1, 1), (20, 1 << 24, 4),
                                            (20, 1 << 31, 4), (4, 1 << 30, 2), (5, 1 << 30, 4)])
def test_one_word_out_of_step(tree, word, flip, want):
    n, leaf, t = tree
    at = int(np.argmax((leaf > 0).any(1) & (n[:, 3] >> 24 > 0)))  # a node with leaves and inner children
    bad = n.copy()
    bad[at, word] ^= np.uint32(flip)
    assert bits(bad, t) == want


@pytest.mark.parametrize("change", ["missing", "extra", "offset"])
def test_leaf_word_and_slots(tree, change):
    n, leaf, t = tree
    bad = n.copy()
    if change == "missing":  # a leaf slot's bits gone
        at, slot = np.argwhere(leaf == 1)[0]
        bad[at, 20] &= ~np.uint32(7 << (3 * slot))
    elif change == "extra":  # bits for an inner or empty slot
        at, slot = np.argwhere(leaf == 0)[0]
        bad[at, 20] |= np.uint32(1 << (3 * slot))
    else:  # a slot's offset that is not its rank
        at, slot = np.argwhere(leaf > 0)[0]
        m = bad[at, 6:8].view(np.uint8)
        m[slot] ^= 1
    assert bits(bad, t) == 4


def test_triangle_ids(tree):
    n, _, t = tree
    bad = t.copy()
    bad[0, 3] = bad[1, 3]
    assert bits(n, bad) == 8
