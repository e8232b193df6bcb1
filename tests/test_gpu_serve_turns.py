"""Small jobs that arrive at every step: each is through in about the steps
its own passes take, however many come after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
N, C, JOBS = 5, 0.6, 48


def _submit(sv, seed, n=N, c=C, pert=0.1):
    import omega_h_v1_b200 as G
    coords, conn, _ = G.box(n, seed, pert)
    return sv.submit(coords, conn, np.full(coords.size // 3, c / n))


def _steps_alone(seed, **kw):
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    _submit(sv, seed, **kw)
    steps = 1
    while sv.step():
        steps += 1
    sv.close()
    return steps


def test_a_job_does_not_wait_for_later_arrivals():
    import omega_h_v1_b200 as G
    alone = max(_steps_alone(s) for s in range(4))
    sv = G.Server(*ARGS, 8 << 30)
    came, took, step = {}, {}, 0

    def stepped():
        left = sv.step()
        for j in sv.poll():
            took[j] = step - came[j] + 1
        return left
    while step < JOBS:
        step += 1
        came[_submit(sv, step)] = step
        stepped()
    arrived = dict(took)   # those that were through before the last one came
    step += 1
    while stepped():
        step += 1
    assert len(took) == JOBS
    sv.close()
    assert max(took.values()) <= alone + 1, (alone, took)
    assert len(arrived) >= JOBS - alone - 1


def test_a_job_does_not_wait_for_a_slow_one():
    import omega_h_v1_b200 as G
    alone = _steps_alone(0, n=6, c=1.0)
    sv = G.Server(*ARGS, 8 << 30)
    a = _submit(sv, 0, n=6, c=1.0)
    b = _submit(sv, 1, n=6, c=1.0, pert=0.3)   # as many passes as a job may take
    for _ in range(alone):
        sv.step()
    assert sv.job_info(a)["finished"] and not sv.job_info(b)["finished"]
    sv.close()
