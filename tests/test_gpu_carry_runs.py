"""Adjacency carried through passes that change few entities, on meshes whose
entity counts end inside a warp's run of 32 rows (6 to 1296 tets): after a
refinement and a coarsening with every adjacency asked for before, the
upward rows (highs, directions, order), the downward ones and the labels are
the oracle's."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu

PAIRS = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def _ask(m):
    for lo, hi in PAIRS:
        m.up(lo, hi)
        if lo:
            m.down(hi, lo)


def _check(g, o, what):
    from oracle import oracle as O
    errs = O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)
    assert not errs, "%s: %s" % (what, errs[:3])
    for lo, hi in PAIRS:
        for x, y in zip(g.up(lo, hi), o.up(lo, hi)):
            assert np.array_equal(x, y), "%s: up(%d,%d)" % (what, lo, hi)
        if lo:
            assert np.array_equal(g.down(hi, lo), o.down(hi, lo)), (what, hi, lo)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("corner", [0, -1])
def test_few_changes(n, corner):
    from oracle import oracle as O
    g, o = build_gpu(n, seed=n, size=2.0 / n), build_cpu(O.Oracle, n, seed=n, size=2.0 / n)
    nv = g.count(0)
    h = np.full(nv, 2.0 / n)
    h[corner] = 0.05 / n          # only the edges of one corner are too long
    for m in (g, o):
        m.free_tag(0, "adapt_size")
        m.add_field(0, "adapt_size", h)
    _ask(g)
    for p in range(3):
        assert g.refine_by_size(0.05) == o.refine_by_size(0.05)
        _check(g, o, "refine %d" % p)
    for m in (g, o):              # and now they are too short
        m.free_tag(0, "adapt_size")
        m.add_field(0, "adapt_size", np.full(m.count(0), 1.0 / n))
    for p in range(2):
        assert g.coarsen_by_size(0.05, 0.6) == o.coarsen_by_size(0.05, 0.6)
        _check(g, o, "coarsen %d" % p)
