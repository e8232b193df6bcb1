"""The server's budget while a union holds a job that has already been handed
back: its bytes stay reserved until the union is gone, and a job that waits
for them gets them soon after, not only once the union's last job is through."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = (1 / 3., 0.3, 4, 50)
SHORT, LONG = (6, 1.0, 0.1), (6, 1.0, 0.3)   # few passes; as many as a job may take


def _submit(sv, job, seed):
    import omega_h_v1_b200 as G
    n, c, pert = job
    coords, conn, _ = G.box(n, seed, pert)
    return sv.submit(coords, conn, np.full(coords.size // 3, c / n))


def _until(sv, job):
    for _ in range(60):
        sv.step()
        if job in sv.poll():
            return
    raise AssertionError("job %d not through" % job)


def test_a_handed_back_job_stays_reserved_while_its_union_holds_it():
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    a, b = _submit(sv, SHORT, 0), _submit(sv, LONG, 1)
    sv.step()
    both = sv.stats()["reserved"]
    _until(sv, a)
    sv.take(a).close()
    assert not sv.job_info(b)["finished"]
    assert sv.stats()["reserved"] == both
    sv.step()
    assert sv.stats()["reserved"] == both
    _until(sv, b)
    assert sv.stats()["reserved"] == 0
    sv.close()


def test_a_waiting_job_gets_the_room_of_one_that_left():
    import omega_h_v1_b200 as G
    sv = G.Server(*ARGS, 8 << 30)
    a, b = _submit(sv, SHORT, 0), _submit(sv, LONG, 1)
    sv.step()
    budget = int(sv.stats()["reserved"])
    sv.close()
    sv = G.Server(*ARGS, budget)
    a, b, c = _submit(sv, SHORT, 0), _submit(sv, LONG, 1), _submit(sv, SHORT, 0)
    sv.step()
    assert sv.stats()["active"] == 2 and sv.stats()["queued"] == 1
    _until(sv, a)
    for _ in range(2):
        assert sv.stats()["reserved"] <= budget
        sv.step()
    assert sv.stats()["queued"] == 0 and sv.stats()["reserved"] <= budget
    assert not sv.job_info(b)["finished"]
    while sv.step():
        assert sv.stats()["reserved"] <= budget
    assert sv.take(c).digest() == sv.take(a).digest()
    sv.close()
