"""Noise does not choose between launch shapes that launch the same kernel the same
way."""
import pytest

from cbc_b200 import autotune
from cbc_b200.autotune import DEFAULT


@pytest.mark.parametrize("lin", ["richardson", "lu"])
@pytest.mark.parametrize("K", [1, 2, 8, 11, 16, 17, 20, 32])
def test_same_launches_are_measured_once(K, lin):
    seen = []

    def measure(cfg):
        seen.append(cfg)
        return 1000.0 + 100.0 * len(seen)        # every later candidate looks faster

    res = autotune.tune_k(K, measure, repeats=1, lin_solver=lin)
    shapes = [autotune.launch_shape(K, c, lin) for c in seen]
    assert len(set(shapes)) == len(shapes)
    assert {autotune.launch_shape(K, c, lin) for c in autotune.candidates(K)} == set(shapes)
    assert seen[0] == DEFAULT
    if lin == "richardson" and K > 16:
        assert res["config"] == DEFAULT and len(seen) == 1
    if lin == "richardson" and K == 1:
        assert all(c.min_blocks == 0 for c in seen)
    if lin == "lu" or 1 < K <= 16:
        assert len(seen) == len(autotune.candidates(K))
