"""Clones of meshes whose arrays end inside a 16-byte word, fill more than
one launch of copies, or are larger than one sweep of its grid."""
import numpy as np
import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extra", [(1, 0), (2, 12), (3, 20), (40, 1)])
def test_clone_is_equal(n, extra):
    import omega_h_v1_b200 as G
    g = build_gpu(n, seed=n)
    rng = np.random.default_rng(n)
    kinds = [(G.T_U8, 1), (G.T_U8, 3), (G.T_U32, 1), (G.T_U64, 1), (G.T_F64, 2)]
    for i in range(extra):
        ty, nc = kinds[i % len(kinds)]
        d = i % 4
        g.add_tag(d, "t%d" % i, rng.integers(0, 200, g.count(d) * nc), ty, nc)
    c = g.clone()
    assert c.digest() == g.digest()
    a, b = c.snapshot(), g.snapshot()
    for d in range(4):
        for x, y in zip(a.tags[d], b.tags[d]):
            assert (x.name, x.type, x.ncomps) == (y.name, y.type, y.ncomps)
            assert np.array_equal(x.data, y.data), (d, x.name)
