"""A coarsening and a swapping pass's build, every dimension of it in one
launch: on boxes that fill no block, part of one and many (where the copies of
wide rows and of short lists take turns), with element fields, and on a mesh
of elements only: the meshes are the oracle's."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


def _same(g, o):
    from oracle import oracle as O
    assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)


@pytest.mark.parametrize("fields", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 12, 20])
def test_full_meshes(n, fields):
    from oracle import oracle as O
    kw = dict(seed=n, pert=0.3, size=2.5 / n, fields=fields)
    g, o = build_gpu(n, **kw), build_cpu(O.Oracle, n, **kw)
    for _ in range(2):
        assert g.coarsen_by_size(0.1, 0.5) == o.coarsen_by_size(0.1, 0.5)
        _same(g, o)
        assert g.swap_slivers(0.6, 1) == o.swap_slivers(0.6, 1)
        _same(g, o)


@pytest.mark.parametrize("n", [2, 5, 12])
def test_elements_only(n):
    import omega_h_v1_b200 as G
    from oracle import oracle as O
    x, conn, _ = G.box(n, n, 0.3)
    g, o = G.Mesh.reduced(3, x, conn), O.Oracle(3, x, conn)
    for m in (g, o):   # swapping asks for the edges' classes: all interior
        m.add_tag(1, "class_dim", np.full(m.count(1), 3, np.uint32), O.T_U32)
    assert g.swap_slivers(0.6, 1) == o.swap_slivers(0.6, 1)
    assert np.array_equal(g.down(3, 0), o.down(3, 0))
