"""Drawing query configurations ends on a scene that has no free one, and
goes on over draws without a free configuration otherwise."""
import numpy as np
import pytest

from gpuprm_b200 import planner, scenes


class Checker:
    """Codes of the n-th call: free[n] free configurations, the rest colliding."""

    def __init__(self, free, most):
        self.free, self.most, self.calls = free, most, 0

    def check_configs(self, q):
        self.calls += 1
        assert self.calls <= self.most, "still drawing"
        codes = np.ones(len(q), np.int32)
        codes[:self.free(self.calls)] = 0
        return codes


def test_a_scene_without_free_configurations_is_refused(monkeypatch):
    monkeypatch.setattr(planner, "QUERY_DRAWS", 4000, raising=False)
    sc = scenes.make_box4(0)
    with pytest.raises(ValueError, match="no free configuration"):
        planner.make_queries(Checker(lambda c: 0, 60), sc, 10, 3)     # 80 configurations a draw


def test_draws_without_a_free_configuration_are_passed_over(monkeypatch):
    monkeypatch.setattr(planner, "QUERY_DRAWS", 400, raising=False)
    sc = scenes.make_box4(0)
    cs = Checker(lambda c: 1 if c % 4 == 0 else 0, 100)               # every fourth draw has one
    a, b = planner.make_queries(cs, sc, 10, 3)
    assert a.shape == b.shape == (10, 4) and cs.calls == 80
    want = np.stack([scenes.uniform_configs(sc, 80, 3 + 424242 + s)[0] for s in range(3, 80, 4)])
    np.testing.assert_array_equal(np.concatenate([a, b]), want)
