"""Qualities of listed edges by as many lanes an edge as the grid has for
each: lists of a few edges (16 lanes), of some ten thousands (fewer) and past
the grid (a thread an edge), with edges that pass the floor and edges that do
not, by one refinement pass: the mesh is the oracle's."""
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,floor", [(1, 0.05), (4, 0.3), (12, 0.25), (18, 0.05), (18, 0.3), (26, 0.25),
                                     (32, 0.25)])
def test_refined_by_any_number_of_lanes(n, floor):
    from oracle import oracle as O
    # about half the edges are longer than the size field asks for
    kw = dict(seed=n, pert=0.2, radial=(0.8 / n, 1.2 / n))
    g, o = build_gpu(n, **kw), build_cpu(O.Oracle, n, **kw)
    assert g.refine_by_size(floor) == o.refine_by_size(floor)
    assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)
