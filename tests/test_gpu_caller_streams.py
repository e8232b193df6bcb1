"""A stream of the caller's: what the library keeps for it goes with the last
mesh on it (the scans' scratch with osh_b200_release_stream), so nothing of
size stays behind a handle that the driver may hand out again."""
import ctypes as C

import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)


def _kept():
    """Bytes the library keeps for its next allocations: what the device's
    memory pool has in use, less what the library counts as in use."""
    import omega_h_v1_b200 as G
    rt = C.CDLL("libcudart.so.12")
    pool, used = C.c_void_p(), C.c_ulonglong()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(used)) == 0   # UsedMemCurrent
    return used.value - G.pool_stats()["used"]


@pytest.mark.parametrize("moved", [False, True])
def test_blocks_go_with_the_last_mesh(moved):
    import torch
    import omega_h_v1_b200 as G
    L = G.lib()
    want = build_gpu(8, seed=1, size=0.7 / 8)
    want.adapt(*ARGS)
    want = want.digest()        # (what it takes on its stream is kept from here on)
    base = build_gpu(8, seed=1, size=0.7 / 8)
    st = torch.cuda.Stream()
    a, b = base.clone(), base.clone()
    torch.cuda.synchronize()
    before = _kept()
    for m in (a, b):
        L.osh_b200_set_stream(m.h, C.c_void_p(st.cuda_stream))
        G.check()
    a.adapt(*ARGS)
    assert a.digest() == want
    a.close()
    assert _kept() > before     # b is still on the stream
    b.adapt(*ARGS)
    assert b.digest() == want
    if moved:
        L.osh_b200_set_stream(b.h, C.c_void_p(0))
        G.check()
        assert _kept() <= before
    b.close()
    if not moved:
        assert _kept() <= before
    L.osh_b200_release_stream(C.c_void_p(st.cuda_stream))
