"""Independent sets at the sizes where their launch changes (one cluster of
blocks up to 8192 entities; lists with and without eight lanes to an entity),
with every edge or few of them candidates, with ties everywhere (unperturbed
boxes), and with dependency chains up to and past the reference's 100 rounds."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pert", [0.0, 0.15])
@pytest.mark.parametrize("n,c", [(2, 0.5), (10, 0.4), (10, 1.35), (11, 0.4), (11, 1.35),
                                 (16, 0.4), (16, 1.62)])
def test_sets_match_oracle(n, c, pert):
    """7930 edges at n = 10, 10,439 at n = 11; c n edges long: all of them at
    0.4, the boxes' diagonals at the larger ones."""
    from oracle import oracle as O
    kw = dict(seed=n, pert=pert, size=c / n)
    g, o = build_gpu(n, **kw), build_cpu(O.Oracle, n, **kw)
    sg, so = g.refine_sets(0.0), o.refine_sets(0.0)
    for k in so:
        assert np.array_equal(sg[k], so[k]), k
    assert so["indset"].any()
    for floor in (0.9, 5.0):   # few and all edges short
        cg, co = g.coarsen_sets(0.05, floor), o.coarsen_sets(0.05, floor)
        for k in co:
            assert np.array_equal(cg[k], co[k]), (floor, k)
    assert g.refine_by_size(0.0) == o.refine_by_size(0.0) == 1
    assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)


def _strip(n):
    """n triangles in a strip whose rungs are the only edges longer than the
    size field, each better than the next: a chain of n + 1 candidates."""
    i = np.arange(n + 2)
    x = np.zeros((n + 2, 3))
    x[:, 0] = np.cumsum(0.5 + 0.5 * i / n)
    x[1::2, 1] = 3.0
    k = np.arange(n)
    t = np.stack([k, k + 1, k + 2], 1)
    t[0::2] = t[0::2][:, [0, 2, 1]]
    return x.ravel(), t.astype(np.uint32).ravel()


def _both(n):
    import omega_h_v1_b200 as G
    from oracle import oracle as O
    x, t = _strip(n)
    out = []
    for m in (G.Mesh.reduced(2, x, t), O.Oracle(2, x, t)):
        m.derive_model_full()
        m.add_field(0, "adapt_size", np.full(n + 2, 2.5))
        out.append(m)
    return out


@pytest.mark.parametrize("n", [7, 40, 60])
def test_chain(n):
    from oracle import oracle as O
    g, o = _both(n)
    assert g.refine_by_size(0.0) == o.refine_by_size(0.0) == 1
    assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)


@pytest.mark.parametrize("n", [120, 1000, 20000])
def test_chain_past_the_cap(n):
    """The pass reports that the set did not settle, leaves the mesh as it
    was, and the device goes on."""
    import omega_h_v1_b200 as G
    x, t = _strip(n)
    g = G.Mesh.reduced(2, x, t)
    g.derive_model_full()
    g.add_field(0, "adapt_size", np.full(n + 2, 2.5))
    before = g.digest()
    for _ in range(2):
        with pytest.raises(G.OshError) as e:
            g.refine_by_size(0.0)
        assert e.value.code == 2   # OSH_B200_E_NOCONVERGE
        assert g.digest() == before
    test_chain(40)
