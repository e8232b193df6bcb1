"""The exclusive scan where its words, chunks, tiles and tile shapes end (a
word is 4 items, a chunk 128, a tile 4096 or, from 4M items on, 8192), with
arrays that start on 16 bytes and arrays that do not, and 32-bit wrap-around.
Whole numbers: exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 3, 4, 5, 127, 128, 129, 511, 513, 4095, 4096, 4097, 8193, 12289]
LONG = [(4 << 20) - 1, 4 << 20, (4 << 20) + 1, (4 << 20) + 8192 * 40 + 7]


@pytest.mark.parametrize("shift_in,shift_out", [(0, 0), (1, 0), (0, 3), (2, 1)])
@pytest.mark.parametrize("n", EDGES + LONG)
def test_exscan(n, shift_in, shift_out):
    import torch
    import omega_h_v1_b200 as G
    rng = np.random.default_rng(n + shift_in)
    a = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    src = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    dst = torch.full((n + 9,), -7, dtype=torch.int32, device="cuda")
    src[shift_in:shift_in + n] = torch.from_numpy(a.view(np.int32)).cuda()
    for _ in range(2):  # the second finds the scratch as the first left it
        rc = G.lib().osh_b200_exscan_u32(C.c_void_p(src.data_ptr() + 4 * shift_in),
                                         C.c_void_p(dst.data_ptr() + 4 * shift_out), n,
                                         C.c_void_p(0), 1)
        assert rc == 0
    out = dst.cpu().numpy().view(np.uint32)
    want = np.zeros(n + 1, np.uint32)
    want[1:] = np.cumsum(a, dtype=np.uint64).astype(np.uint32)  # (integer wrap-around)
    assert np.array_equal(out[shift_out:shift_out + n + 1], want)
    assert (dst.cpu().numpy()[shift_out + n + 1:] == -7).all()
    assert (dst.cpu().numpy()[:shift_out] == -7).all()
