"""bench.py's check of its many-mesh legs: which meshes differ, in which leg,
and a line that says so does not pass for a good one."""
import bench


def test_differing_meshes():
    plain = {0: 11, 1: 12, 2: 13}
    assert bench.differing_meshes(plain, {"a": dict(plain), "b": dict(plain)}) == []
    assert bench.differing_meshes(plain, {"b": {0: 11, 1: 12}, "a": {0: 11, 1: 9, 2: 13}}) == [
        ("a", 1), ("b", 2)]


def test_all_identical():
    good = {"value": 1.0, "fp32_filter": {"identical_to_plain": True},
            "batched_cfg4": {"identical_to_plain": True, "legs": {"x": 2.0}}}
    assert bench.all_identical(good)
    for bad in (False, None):
        assert not bench.all_identical(dict(good, batched_cfg4={"identical_to_plain": bad}))
    assert not bench.all_identical({"identical_concurrent": False})
