"""Element gradients and their recovery at the sizes and component counts
where the kernels' blocks and batches end: one block and less, a ragged last
block, rows shorter than a batch, counts with and without a kernel of their
own, triangles and tets. Bit-identical to the oracle."""
import numpy as np
import pytest

from conftest import build_cpu, build_gpu

pytestmark = pytest.mark.gpu


def _pair(dim, n):
    from oracle import oracle as O
    import omega_h_v1_b200 as G
    if dim == 3:
        return build_gpu(n, size=1.0), build_cpu(O.Oracle, n, size=1.0)
    j, i = np.divmod(np.arange((n + 1) * (n + 1)), n + 1)
    x = np.stack([i / n, j / n + 0.1 * np.sin(i), 0.0 * i], axis=1).ravel()
    v = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    conn = np.stack([v, v + 1, v + n + 2, v + n + 2, v + n + 1, v], axis=1)
    conn = conn.astype(np.uint32).ravel()
    g, o = G.Mesh.reduced(2, x, conn), O.Oracle(2, x, conn)
    g.derive_model_full()
    o.derive_model_full()
    return g, o


@pytest.mark.parametrize("nc", [1, 2, 3, 5])
@pytest.mark.parametrize("dim,n", [(3, 1), (3, 5), (2, 1), (2, 8), (2, 9)])
def test_gradients_and_recovery_match_oracle(dim, n, nc):
    g, o = _pair(dim, n)
    f = np.random.default_rng(100 * n + nc).normal(size=g.count(0) * nc)
    for m in (g, o):
        m.add_field(0, "f", f, nc)
        m.element_gradients("f")
        m.recover_by_volume("grad_f")
    sg, so = g.snapshot(), o.snapshot()
    for d in (dim, 0):
        a, b = sg.tag(d, "grad_f").data, so.tag(d, "grad_f").data
        assert a.size == b.size and np.array_equal(a, b)
