"""Upward adjacency of one word a use: rows sorted in place inside and past
their kernel's network (a hub's row beside short ones), and the highs and
directions taken apart again, for every pair of dimensions: the stable order
of the downward array."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(n):
    """n triangles about vertex 0: its row holds n, the rim's one or two"""
    a = 2 * np.pi * np.arange(n + 1) / (n + 1)
    x = np.zeros((n + 2, 3))
    x[1:, 0], x[1:, 1] = np.cos(a), np.sin(a)
    i = np.arange(n)
    return 2, x.ravel(), np.stack([0 * i, i + 1, i + 2], 1).astype(np.uint32).ravel()


def _ring(n):
    """n tets about the edge (0, 1)"""
    a = 2 * np.pi * np.arange(n) / n
    x = np.zeros((n + 2, 3))
    x[1, 2] = 1.0
    x[2:, 0], x[2:, 1], x[2:, 2] = np.cos(a), np.sin(a), 0.5
    i = np.arange(n)
    return 3, x.ravel(), np.stack([0 * i, i + 2, (i + 1) % n + 2, 0 * i + 1], 1).astype(np.uint32).ravel()


@pytest.mark.parametrize("make", [_fan, _ring])
@pytest.mark.parametrize("n", [3, 8, 9, 31, 33, 64, 65, 127, 1000, 4099])
def test_rows(make, n):
    import omega_h_v1_b200 as G
    dim, x, conn = make(n)
    m = G.Mesh.reduced(dim, x, conn)
    # (deriving the edges of a row past the cap of 256 is refused)
    for low, high in [(0, dim)] + [(l, h) for h in range(1, dim + 1) for l in range(h)] * (n < 256):
        lows = m.down(high, low)
        lph = lows.size // m.count(high)
        want = np.argsort(lows, kind="stable")
        offs, adj, dirs = m.up(low, high)
        assert np.array_equal(np.diff(offs), np.bincount(lows, minlength=m.count(low)))
        assert np.array_equal(adj, want // lph)
        assert np.array_equal(dirs, want % lph)
