"""Boxes whose perturbation inverts elements, against the oracle, and two
inputs of the independent set in which an entity would wait for itself or two
for each other: an edge of one vertex (swaps in a tangled mesh leave such
edges) and global numbers given twice."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu
from test_gpu_capi import _mesh_from_snapshot

pytestmark = pytest.mark.gpu


# (whose passes leave nothing twice and no edge of one vertex)
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
    """No vertex is its own neighbour. (The sets alone: no pass is run.)"""
    import omega_h_v1_b200 as G
    base = build_gpu(4, seed=1, size=3.0 / 4)
    s = base.snapshot()
    v = int(np.flatnonzero(s.tag(0, "class_dim").data == 3)[0])
    s.conn[1] = np.append(s.conn[1], [v, v]).astype(np.uint32)
    for t in s.tags[1]:
        like = s.tag(0, t.name).data[v]
        t.data = np.append(t.data, like).astype(t.data.dtype)
    s.counts[1] += 1
    m = _mesh_from_snapshot(G, s)
    sets = m.coarsen_sets(0.0, 1 / 3.)
    ind, cand, edges = sets["indset"], sets["candidates"], m.down(1, 0).reshape(-1, 2)
    a, b = edges[edges[:, 0] != edges[:, 1]].T
    # independent, and no candidate is left out without a neighbour in the set
    assert not (ind[a] & ind[b]).any()
    near = np.zeros(m.count(0), bool)
    near[a[ind[b] == 1]] = True
    near[b[ind[a] == 1]] = True
    assert cand[v] and ind[v]      # (its quality, no element left to judge, is the best there is)
    assert (ind[cand == 1] | near[cand == 1]).all()


def test_global_numbers_given_twice():
    """They leave ties of equal qualities open; the set is settled by index."""
    m = build_gpu(8, pert=0, size=5.0 / 8, parallel=True)   # (exact coordinates: ties everywhere)
    for d in range(4):
        m.set_globals(d, np.zeros(m.count(d), np.uint64))
    sets = m.coarsen_sets(0.0, 1 / 3.)
    ind, cand, edges = sets["indset"], sets["candidates"], m.down(1, 0).reshape(-1, 2)
    a, b = edges.T
    assert not (ind[a] & ind[b]).any()
    near = np.zeros(m.count(0), bool)
    near[a[ind[b] == 1]] = True
    near[b[ind[a] == 1]] = True
    assert cand.any() and (ind[cand == 1] | near[cand == 1]).all()
