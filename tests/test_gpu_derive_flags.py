"""The flags of a derivation that stay zero between uses: a refusal (a row past
the cap, met by the star, the dual or the derivation of a model) leaves them so
-- asked again it is refused again, and the next mesh of the same stream and
of the same mailbox derives as the oracle."""
import numpy as np
import pytest

from test_gpu_star_dual import _ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["star", "dual", "derive", "edges"])
def test_refused_then_derived(first):
    import omega_h_v1_b200 as G
    from oracle import oracle as O
    g = G.Mesh.reduced(3, *_ring(300, True))
    ask = {"star": lambda: g.star(0, 3), "dual": g.dual, "derive": g.derive_model_full,
           "edges": lambda: g.down(1, 0)}[first]
    for _ in range(2):
        with pytest.raises(G.OshError) as e:
            ask()
        assert e.value.code == 4   # OSH_B200_E_ARG
    del g
    for n in (3, 64):
        x, conn = _ring(n, True)
        g, o = G.Mesh.reduced(3, x, conn), O.Oracle(3, x, conn)
        g.derive_model_full()
        o.derive_model_full()
        assert not O.mesh_diff(g.snapshot(), o.snapshot(), rel_tol=0.0)


@pytest.mark.parametrize("n", [1, 4])
def test_up_counts_return_to_zero(n):
    """rows of one pair after another on one stream, from the same counts"""
    import omega_h_v1_b200 as G
    for k in (4 * n, n):
        x, conn, _ = G.box(k, k, 0.1)
        m = G.Mesh.reduced(3, x, conn)
        for low, high in ((0, 3), (0, 1), (1, 2), (0, 2), (2, 3), (1, 3)):
            lows = m.down(high, low)
            want = np.argsort(lows, kind="stable")
            offs, adj, dirs = m.up(low, high)
            lph = lows.size // m.count(high)
            assert np.array_equal(adj, want // lph) and np.array_equal(dirs, want % lph)


def test_up_counts_of_threads_on_one_stream():
    """host threads that build rows of their own meshes on the same stream"""
    import threading
    import omega_h_v1_b200 as G

    def work(k, out):
        x, conn, _ = G.box(k, k, 0.1)
        lows = conn.reshape(-1)
        want = np.argsort(lows, kind="stable")
        ok = True
        for _ in range(20):
            m = G.Mesh.reduced(3, x, conn)
            offs, adj, dirs = m.up(0, 3)
            ok = ok and np.array_equal(adj, want // 4) and np.array_equal(dirs, want % 4)
        out.append(ok)

    out = []
    ts = [threading.Thread(target=work, args=(k, out)) for k in (3, 5, 8, 12)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert out == [True] * 4
