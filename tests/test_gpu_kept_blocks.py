"""Device blocks, streams and mailboxes that meshes give back and others
take: the memory in use goes back to what it was, a released stream keeps
nothing, and meshes made, adapted, moved between streams and freed by several
threads at once end as they do alone."""
import threading

import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)


def _adapted(n, seed):
    m = build_gpu(n, seed=seed, size=0.7 / n)
    m.adapt(*ARGS)
    return m


def test_memory_in_use_returns():
    import torch
    import omega_h_v1_b200 as G
    _adapted(6, 0).close()
    torch.cuda.synchronize()
    before = G.pool_stats()["used"]
    for i in range(3):
        ms = [_adapted(n, i) for n in (3, 6, 10)]
        assert G.pool_stats()["used"] > before
        for m in ms:
            m.close()
    torch.cuda.synchronize()
    # (scratch that streams keep may have grown with the meshes)
    assert G.pool_stats()["used"] <= before + (4 << 20)


def test_moved_between_streams():
    import torch
    import omega_h_v1_b200 as G
    L = G.lib()
    want = _adapted(5, 1).digest()
    for _ in range(3):
        m = build_gpu(5, seed=1, size=0.7 / 5)
        other = build_gpu(4, seed=2, size=0.7 / 4)
        st = torch.cuda.Stream()
        for x, s in ((m, st.cuda_stream), (other, 0)):
            L.osh_b200_set_stream(x.h, G.C.c_void_p(s))
        c = m.clone()
        m.adapt(*ARGS)
        other.adapt(*ARGS)
        L.osh_b200_set_stream(m.h, G.C.c_void_p(0))
        L.osh_b200_release_stream(G.C.c_void_p(st.cuda_stream))
        G.check()
        c.adapt(*ARGS)
        assert m.digest() == want and c.digest() == want


def test_threads():
    want = {n: _adapted(n, n).digest() for n in (3, 4, 5, 6)}
    bad = []

    def work(k):
        try:
            for i in range(6):
                n = 3 + (k + i) % 4
                m = build_gpu(n, seed=n, size=0.7 / n)
                c = m.clone()
                m.close()
                c.adapt(*ARGS)
                if c.digest() != want[n]:
                    bad.append((k, i, n))
                c.close()
        except Exception as e:   # reported by the assertion below
            bad.append(repr(e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
