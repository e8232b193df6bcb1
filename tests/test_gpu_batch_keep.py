"""Unions kept between passes: meshes that end at different passes, a union
regathered because most of its elements wait, one split because it outgrew
its limit, and jobs that join a server while a kept union runs. Every mesh
ends as it does alone."""
import numpy as np
import pytest

from conftest import build_gpu

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)


def _alone(kw):
    m = build_gpu(**kw)
    m.adapt(*ARGS)
    return m.digest()


@pytest.mark.parametrize("cases,limit", [
    # ends at different passes; nothing to do at all for two of them
    ([dict(n=4, size=0.4 / 4), dict(n=2, size=0.6), dict(n=5, size=0.16), dict(n=3, size=1 / 3.),
      dict(n=6, size=3.0 / 6)], 0),
    # over a million elements wait for a few thousand
    ([dict(n=58, size=1.25 / 58), dict(n=4, size=0.45 / 4), dict(n=5, size=0.5 / 5)], 0),
    # the union outgrows its limit and is gathered in smaller ones
    ([dict(n=5, size=0.5 / 5), dict(n=4, size=0.4 / 4), dict(n=6, size=0.8 / 6)], 2500),
])
def test_batch_with_kept_unions(cases, limit):
    import omega_h_v1_b200 as G
    ms = [build_gpu(seed=i, **kw) for i, kw in enumerate(cases)]
    changed, status, stats = G.adapt_batch(ms, *ARGS, max_union_elems=limit)
    assert not any(status)
    want = [_alone(dict(kw, seed=i)) for i, kw in enumerate(cases)]
    assert [m.digest() for m in ms] == want


def test_jobs_join_a_kept_union():
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    jobs, ids = [], []
    for i, (n, c) in enumerate([(4, 0.5), (5, 0.6), (3, 1.0), (4, 0.8), (6, 0.9)]):
        coords, conn, _ = G.box(n, i, 0.1)
        jobs.append((n, c))
        ids.append(sv.submit(coords, conn, np.full(coords.size // 3, c / n)))
        sv.step()                      # earlier jobs are already under way
    while sv.step():
        pass
    for i, (n, c) in enumerate(jobs):
        got = sv.take(ids[i]).snapshot()
        alone = build_gpu(n, seed=i, size=c / n)
        alone.adapt(*ARGS)
        want = alone.snapshot()
        assert got.counts == want.counts
        for d in range(1, 4):
            assert np.array_equal(got.conn[d], want.conn[d])
        assert np.array_equal(got.tag(0, "coordinates").data, want.tag(0, "coordinates").data)
    sv.close()
