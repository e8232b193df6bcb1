"""Vertex stars and element duals of meshes that hold elements only, on rings
of tets about an edge (the edge's vertices have a neighbour or an element per
tet: rows that end inside a warp's step, and past the cap of 256) and on
boxes: the oracle's, in its order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(n, closed):
    """n tets about the edge (0, 1), between n (closed) or n + 1 vertices"""
    nr = n if closed else n + 1
    a = 2 * np.pi * np.arange(nr) / (n + 1)
    x = np.zeros((nr + 2, 3))
    x[1, 2] = 1.0
    x[2:, 0], x[2:, 1], x[2:, 2] = np.cos(a), np.sin(a), 0.5
    i = np.arange(n)
    conn = np.stack([0 * i, i + 2, (i + 1) % nr + 2, 0 * i + 1], 1).astype(np.uint32)
    return x.ravel(), conn.ravel()


def _pair(x, conn):
    import omega_h_v1_b200 as G
    from oracle import oracle as O
    return G.Mesh.reduced(3, x, conn), O.Oracle(3, x, conn)


@pytest.mark.parametrize("n,closed", [(1, False), (3, True), (8, False), (30, True), (31, False),
                                      (64, True), (253, True)])
def test_ring(n, closed):
    g, o = _pair(*_ring(n, closed))
    for a, b in zip(g.star(0, 3), o.star(0, 3)):
        assert np.array_equal(a, b)
    assert np.array_equal(g.dual(), o.dual())
    g, o = _pair(*_ring(n, closed))
    g.derive_model_full()
    o.derive_model_full()
    from oracle import oracle as O
    assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)


@pytest.mark.parametrize("n", [1, 3, 6])
def test_box(n):
    import omega_h_v1_b200 as G
    x, conn, _ = G.box(n, n, 0.2)
    g, o = _pair(x, conn)
    assert np.array_equal(g.dual(), o.dual())
    for a, b in zip(g.star(0, 3), o.star(0, 3)):
        assert np.array_equal(a, b)


def test_rows_past_the_cap_are_refused():
    import omega_h_v1_b200 as G
    g = G.Mesh.reduced(3, *_ring(300, True))
    for f in (lambda: g.star(0, 3), g.dual):
        with pytest.raises(G.OshError) as e:
            f()
        assert e.value.code == 4   # OSH_B200_E_ARG
