"""Every tile shape that the tuning table can name for the scans, at sizes
around that shape's own tiles, and the shape that long scans take instead.
Whole numbers: exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = 4 << 20          # from here on a scan with 16 items a thread takes 256 x 32


@pytest.fixture
def shape(request):
    import omega_h_v1_b200 as G
    L, was = G.lib(), {}
    for name, value in zip((b"scan_threads", b"scan_items"), request.param):
        old = C.c_uint()
        assert L.osh_b200_tuning_get(name, C.byref(old)) == 0
        was[name] = old.value
        assert L.osh_b200_tuning_set(name, value) == 0
    yield request.param
    for name, value in was.items():
        assert L.osh_b200_tuning_set(name, value) == 0


@pytest.mark.parametrize("shape", [(t, i) for t in (256, 512) for i in (8, 16)], indirect=True)
def test_around_the_tiles(shape):
    import torch
    import omega_h_v1_b200 as G
    tile = shape[0] * shape[1]
    sizes = [k * tile + d for k in (1, 2, 3, 33) for d in (-1, 0, 1)] + [128, tile // 2 + 5]
    sizes += [LONG + d for d in (-1, 0, 1)] + [LONG + 8192 + d for d in (-1, 0, 1)]
    a = np.random.default_rng(tile).integers(0, 1 << 32, max(sizes), dtype=np.uint32)
    want = np.zeros(max(sizes) + 1, np.uint32)
    want[1:] = np.cumsum(a, dtype=np.uint64).astype(np.uint32)
    src, ref = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, want))
    for n in sizes + sizes[::-1]:      # long after short, short after long
        dst = torch.full((n + 2,), -7, dtype=torch.int32, device="cuda")
        rc = G.lib().osh_b200_exscan_u32(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()),
                                         n, C.c_void_p(0), 1)
        assert rc == 0
        assert torch.equal(dst[:n + 1], ref[:n + 1]), n
        assert int(dst[n + 1]) == -7
