"""The per-edge selections where a block's tile of edges ends (boxes of 19 to
1116 edges, a tile being 1024) with some edges selected and some not, with
and without the single-precision filter: the sets and qualities are the
oracle's, the least quality is found wherever it lies, and every edge's
decision is counted once."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("filt", [False, True])
@pytest.mark.parametrize("n", [1, 2, 4, 5])
def test_selections_match_oracle(n, filt):
    import omega_h_v1_b200 as G
    from oracle import oracle as O
    # about half the edges are longer than the size field asks for, and
    # about half shorter than two thirds of it
    kw = dict(seed=n, pert=0.2, radial=(0.8 / n, 1.2 / n))
    g, o = build_gpu(n, **kw), build_cpu(O.Oracle, n, **kw)
    g.set_fp32_filter(filt)
    ne = g.count(1)
    G.fp32_stats(reset=True)
    sg, so = g.refine_sets(0.05), o.refine_sets(0.05)
    for k in so:
        assert np.array_equal(sg[k], so[k]), k
    if n > 1:
        assert 0 < so["candidate"].sum() < ne
    st = G.fp32_stats(reset=True)
    assert st["decided"] + st["rechecked"] >= (ne if filt else 0)
    if not filt:
        assert st["decided"] + st["rechecked"] == 0
    cg, co = g.coarsen_sets(0.05, 2 / 3.), o.coarsen_sets(0.05, 2 / 3.)
    for k in co:
        assert np.array_equal(cg[k], co[k]), k
    assert np.array_equal(g.qualities(), o.qualities())
    assert g.min_quality() == o.min_quality()
