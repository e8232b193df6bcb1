"""A scan whose look-back gave up is reported by the call that issued it, on
whatever stream: E_TIMEOUT, and the next call runs as ever. The give-up is
recorded by the host (osh_b200_selftest_scan_report); no wait runs out."""
import ctypes as C

import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
NS = (4, 5, 16)   # (with size 0.5 / n: 16 is past what concurrent adapts group)


def _meshes():
    return [build_gpu(n, seed=n, size=0.5 / n) for n in NS]


@pytest.fixture(scope="module")
def alone():
    ms = _meshes()
    for m in ms:
        m.adapt(*ARGS)
    return [m.digest() for m in ms]


def _one_by_one(ms):
    for m in ms:
        m.adapt(*ARGS)


def _batch(ms):
    import omega_h_v1_b200 as G
    G.adapt_batch(ms, *ARGS)


def _concurrent(ms):
    import omega_h_v1_b200 as G
    G.adapt_concurrent(ms, *ARGS, nthreads=2)


def _served(ms):
    import numpy as np
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    try:
        for n in NS:
            coords, conn, _ = G.box(n, n, 0.1)
            sv.submit(coords, conn, np.full(coords.size // 3, 0.5 / n))
        while sv.step():
            pass
    finally:
        sv.close()


@pytest.mark.parametrize("nth", [1, 7, 40])
@pytest.mark.parametrize("run", [_one_by_one, _batch, _concurrent, _served])
def test_reported(run, nth, alone):
    import omega_h_v1_b200 as G
    ms = _meshes()
    G.lib().osh_b200_selftest_scan_report(nth)
    try:
        with pytest.raises(G.OshError) as e:
            run(ms)
    finally:
        G.lib().osh_b200_selftest_scan_report(0)
    assert e.value.code == 7
    for m in ms:
        m.close()
    ms = _meshes()
    run(ms)
    if run is not _served:
        assert [m.digest() for m in ms] == alone


def test_reported_when_the_scratch_grows():
    import torch
    import omega_h_v1_b200 as G
    L = G.lib()
    st = torch.cuda.Stream()
    a = torch.ones(20 << 20, dtype=torch.int32, device="cuda")
    o = torch.empty((20 << 20) + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def scan(n, check):
        return L.osh_b200_exscan_u32(C.c_void_p(a.data_ptr()), C.c_void_p(o.data_ptr()), n,
                                     C.c_void_p(st.cuda_stream), check)
    L.osh_b200_selftest_scan_report(1)
    assert scan(100, 0) == 0
    assert scan(20 << 20, 1) == 7      # the scratch of a short scan does not do for it
    L.osh_b200_clear_error()
    assert scan(20 << 20, 1) == 0
    assert int(o[-1]) == 20 << 20
    L.osh_b200_release_stream(C.c_void_p(st.cuda_stream))
