"""Boxes whose perturbation inverts elements. Swaps there can leave an edge
between one vertex and itself, and edges and faces twice, which the later
passes meet: every call ends, and where nothing is there twice, as in the
oracle, whose mesh_adapt goes through such meshes too."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed,size,layers", [(8, 336, 2.313207571603746, 4),
                                                (7, 183, 2.3, 1), (7, 62, 2.6, 4)])
def test_adapt_matches_the_oracle(n, seed, size, layers):
    from oracle import oracle as O
    kw = dict(n=n, seed=seed, pert=0.3, size=size / n)
    m, o = build_gpu(**kw), build_cpu(O.Oracle, **kw)
    assert m.min_quality() < 0
    assert m.adapt(1 / 3., 0.3, layers, 30) == o.adapt(1 / 3., 0.3, layers, 30) == 1
    errs = O.mesh_diff(m.snapshot(), o.snapshot(), rel_tol=1e-12)
    assert not errs, errs[:5]


def test_an_edge_of_one_vertex():
    """Its vertex is no neighbour of its own in the independent set of the
    sliver collapses. (Which of two equal edges is kept is open: the result
    is not compared.)"""
    m = build_gpu(8, seed=336, pert=0.3, size=2.313207571603746 / 8)
    passes = [lambda: m.refine_by_size(m.min_quality()),
              lambda: m.coarsen_by_size(m.min_quality(), 1 / 3.),
              lambda: m.swap_slivers(0.3, 1)]
    for p in passes:
        for _ in range(30):
            if not p():
                break
    ends = m.down(1, 0).reshape(-1, 2)
    assert (ends[:, 0] == ends[:, 1]).any()
    assert m.coarsen_slivers(0.3, 1) == 1


def test_global_numbers_given_twice():
    """They leave ties of equal qualities open; the set is settled by index."""
    m = build_gpu(5, pert=0, size=0.5 / 5, parallel=True)
    for d in range(4):
        m.set_globals(d, np.zeros(m.count(d), np.uint64))
    ind = m.refine_sets(0.0)["indset"]
    assert ind.any()
    edges = m.down(3, 1).reshape(-1, 6)
    assert (ind[edges].sum(axis=1) <= 1).all()     # no two in one tet
