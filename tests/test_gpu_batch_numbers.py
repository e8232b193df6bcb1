"""Global numbers that are not the local indices, in a batch: they break the
ties of equal qualities, so a mesh that waits while others of its batch are
changed must still have its own when its turn comes. Unperturbed boxes, where
ties are everywhere; every mesh ends as it does alone, numbers included."""
import numpy as np
import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
# refined several times over; only coarsened; only shaped (swaps); as they are
CASES = [dict(n=4, pert=0, size=0.5 / 4), dict(n=8, pert=0, size=3.2 / 8),
         dict(n=6, pert=0.3, size=1.1 / 6), dict(n=3, pert=0, size=1.2 / 3),
         dict(n=7, pert=0, size=3.5 / 7), dict(n=5, pert=0.28, size=1.1 / 5)]


def _mesh(i, numbered):
    m = build_gpu(seed=i, parallel=True, **CASES[i])
    if numbered:
        rng = np.random.default_rng(100 + i)
        for d in range(4):
            m.set_globals(d, rng.permutation(m.count(d)).astype(np.uint64))
    return m


# every mesh numbered by its caller, or every second one
@pytest.mark.parametrize("limit", [0, 3000])
@pytest.mark.parametrize("every", [1, 2])
def test_numbers_kept_while_a_mesh_waits(every, limit):
    import omega_h_v1_b200 as G
    alone = [_mesh(i, i % every == 0) for i in range(len(CASES))]
    for m in alone:
        m.adapt(*ARGS)
    ms = [_mesh(i, i % every == 0) for i in range(len(CASES))]
    changed, status, stats = G.adapt_batch(ms, *ARGS, max_union_elems=limit)
    assert not any(status)
    assert [m.digest() for m in ms] == [m.digest() for m in alone]
    for m, a in zip(ms, alone):
        for d in range(4):
            assert np.array_equal(m.globals(d), a.globals(d))
