"""Host threads that issue on one stream, the legacy default one or a
caller's, each with meshes of its own: every mesh ends as it does alone."""
import ctypes as C
import threading

import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
NS = (3, 5, 8, 12)


def _mesh(n):
    return build_gpu(n, seed=n, size=0.7 / n, fields=n == 5)


@pytest.mark.parametrize("callers", [False, True])
def test_threads_on_one_stream(callers):
    import torch
    import omega_h_v1_b200 as G
    L = G.lib()
    want = {}
    for n in NS:
        m = _mesh(n)
        m.adapt(*ARGS)
        want[n] = m.digest()
    st = torch.cuda.Stream()
    handle = C.c_void_p(st.cuda_stream if callers else 0)
    bad = []

    def work(k):
        try:
            for i in range(8):
                n = NS[(k + i) % len(NS)]
                m = _mesh(n)
                L.osh_b200_set_stream(m.h, handle)
                G.check()
                m.adapt(*ARGS)
                if m.digest() != want[n]:
                    bad.append((k, i, n))
                m.close()
        except Exception as e:   # reported by the assertion below
            bad.append(repr(e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
    if callers:
        L.osh_b200_release_stream(handle)
