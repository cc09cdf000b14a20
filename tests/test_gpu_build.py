"""Builder kernels at the sizes where they can go wrong: one triangle, fewer
than a leaf holds, around a warp and a tile of the clustering, and around the
cluster count that the one-block kernel takes over from (4,096).  The tree is
checked on the host: every triangle in exactly one leaf, every child box
containing its subtree's triangles, and its surface-area cost against the cost
of a rebuild of the same triangles in shuffled order (the same algorithm over
the same Morton order: equal up to ties, 2%).  Equal triangles and points on a line
exercise the ties; they merge one pair per iteration, so up to 4,098 of them
make a tree that is refused as too deep for the traversal stack, and more take
the radix tree instead."""
import numpy as np
import pytest

import colvillea_b200 as cb
from colvillea_b200 import scenes

pytestmark = pytest.mark.gpu


def check(nodes, tris):
    """Exact boxes bottom up; returns the triangle ids in leaf order."""
    f = tris.reshape(-1, 3, 4)[:, :, :3]
    seen = np.zeros(len(f), int)
    lo, hi = np.full((len(nodes), 3), np.inf), np.full((len(nodes), 3), -np.inf)
    for i in range(len(nodes) - 1, -1, -1):
        n = nodes[i]
        p = n[:3].view(np.float32).astype(np.float64)
        e = np.array([np.ldexp(1.0, int((n[3] >> (8 * a)) & 255) - 127) for a in range(3)])
        imask, base, tb = int(n[3] >> 24), int(n[4]), int(n[5])
        b = n.view(np.uint8).reshape(-1)
        meta = b[24:32]
        qlo = np.stack([b[32:40], b[40:48], b[48:56]], 1)
        qhi = np.stack([b[56:64], b[64:72], b[72:80]], 1)
        rank = 0
        for s in range(8):
            if (imask >> s) & 1:
                c = base + rank
                rank += 1
                assert i < c < len(nodes)
                l, h = lo[c], hi[c]
            elif meta[s]:
                k = bin(int(meta[s]) >> 5).count("1")
                at = tb + (int(meta[s]) & 31)
                seen[at:at + k] += 1
                l, h = f[at:at + k].min((0, 1)).astype(np.float64), f[at:at + k].max((0, 1)).astype(np.float64)
            else:
                assert (qlo[s] == 255).all() and (qhi[s] == 0).all()
                continue
            assert (p + e * qlo[s] <= l).all() and (p + e * qhi[s] >= h).all()
            lo[i], hi[i] = np.minimum(lo[i], l), np.maximum(hi[i], h)
    assert (seen == 1).all()
    return np.sort(tris[:, 3].view(np.uint32))


def build(verts):
    n = len(verts)
    m = scenes.Mesh(verts.reshape(-1, 3).astype(np.float32), None, np.tile(np.float32([1, 0, 0]), (3 * n, 1)), None,
                    np.arange(3 * n, dtype=np.uint32).reshape(n, 3))
    it = cb.Integrator.createIntegrator(cb.IntegratorType.WavefrontPathTracing, 8, 8)
    it.buildBLAS([m])
    it.buildTLAS([(0, 0, scenes.IDENTITY)])
    out = it.bvh(), it.stats()["bvh_sah_build"]
    it.close()
    return out


@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 31, 33, 255, 1023, 1025, 4095, 4096, 4097, 6000, 20000])
@pytest.mark.parametrize("kind", ["soup", "equal", "line"])
def test_tree(n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-10, 10, (n, 1, 3))
    if kind == "soup":
        v = c + rng.normal(scale=0.2, size=(n, 3, 3))
    elif kind == "equal":
        v = np.tile(rng.normal(size=(1, 3, 3)), (n, 1, 1))
    else:
        v = np.tile(c * [1, 0, 0], (1, 3, 1))
    if (kind == "equal" and 200 <= n <= 4097) or (kind == "line" and 31 <= n <= 4097):
        with pytest.raises(cb.ClError, match="exceeds the traversal stack"):
            build(v)
        return
    (nodes, tris), sah = build(v)
    np.testing.assert_array_equal(check(nodes, tris), np.arange(n))
    if kind == "soup" and n > 1:
        _, again = build(v[rng.permutation(n)])
        assert abs(sah - again) <= 0.02 * sah
