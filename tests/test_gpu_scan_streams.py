"""Scans of mixed sizes issued by several host threads, each on a stream of
its own: a scan finds its stream's scratch as the scan before it left it, a
short one after a long one and the other way round, with the device busy with
the other streams' scans. Whole numbers: exact."""
import ctypes as C
import threading

import numpy as np
import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

# one tile, a few, some hundred and some thousand of them
SIZES = [1, 700, 9000, 70001, 400000, (2 << 20) + 5, (20 << 20) + 3]
THREADS, ROUNDS = 4, 500


def test_mixed_sizes_on_four_streams():
    import torch
    import omega_h_v1_b200 as G
    L = G.lib()
    rng = np.random.default_rng(0)
    src, want = [], []
    for n in SIZES:
        a = rng.integers(0, 1 << 32, n, dtype=np.uint32)
        w = np.zeros(n + 1, np.uint32)
        w[1:] = np.cumsum(a, dtype=np.uint64).astype(np.uint32)
        src.append(torch.from_numpy(a.view(np.int32)).cuda())
        want.append(torch.from_numpy(w.view(np.int32)).cuda())
    torch.cuda.synchronize()
    bad, left = [None] * THREADS, []

    def work(k):
        try:
            torch.cuda.set_device(0)
            order = np.random.default_rng(k + 1)
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                dst = [torch.empty(n + 1, dtype=torch.int32, device="cuda") for n in SIZES]
                wrong = torch.zeros((), dtype=torch.int64, device="cuda")
                for _ in range(ROUNDS):
                    for q in order.choice(len(SIZES), 3, p=[.2, .2, .2, .15, .1, .1, .05]):
                        rc = L.osh_b200_exscan_u32(C.c_void_p(src[q].data_ptr()),
                                                   C.c_void_p(dst[q].data_ptr()), SIZES[q],
                                                   C.c_void_p(st.cuda_stream), 0)
                        assert rc == 0
                        wrong += (dst[q] != want[q]).sum()
                rc = L.osh_b200_exscan_u32(C.c_void_p(src[0].data_ptr()),
                                           C.c_void_p(dst[0].data_ptr()), SIZES[0],
                                           C.c_void_p(st.cuda_stream), 1)
                assert rc == 0
                st.synchronize()
                bad[k] = int(wrong)
            L.osh_b200_release_stream(C.c_void_p(st.cuda_stream))
        except Exception as e:   # reported by the assertion below
            left.append(repr(e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not left, left
    assert bad == [0] * THREADS


def test_meshes_of_many_tiles_on_four_streams():
    """Adapts whose scans have tens of tiles, side by side: each as alone."""
    import omega_h_v1_b200 as G
    args = (1 / 3., 0.3, 4, 50)
    cases = [dict(n=n, seed=n, size=1.0 / n) for n in (32, 30, 28, 26, 24, 22, 20, 18)]
    base = [build_gpu(**kw) for kw in cases]
    want = []
    for m in base:
        c = m.clone()
        c.adapt(*args)
        want.append(c.digest())
        c.close()
    for _ in range(5):
        ms = [m.clone() for m in base]
        _, status, _ = G.adapt_concurrent(ms, *args, nthreads=4)
        assert not any(status)
        assert [m.digest() for m in ms] == want
        for m in ms:
            m.close()
