"""Small jobs that arrive at every step: each is through in about the steps
its own passes take, however many come after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
N, C, JOBS = 5, 0.6, 48


def _submit(sv, seed):
    import omega_h_v1_b200 as G
    coords, conn, _ = G.box(N, seed, 0.1)
    return sv.submit(coords, conn, np.full(coords.size // 3, C / N))


def _steps_alone(seed):
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    _submit(sv, seed)
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
    # a union's members are through a point of the loop together, and those
    # that join it do so before its first member is past refinement
    assert max(took.values()) <= 2 * alone + 2, (alone, took)
    assert len(arrived) >= JOBS - 2 * alone - 2
