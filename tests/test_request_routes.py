"""Which kernels a request takes: one launch for a small one, the large
kernels' launches where the caller has set a launch shape, an edge split or
the per-kernel profile, with the same codes."""
import numpy as np
import pytest

from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FP64_BAND
from gpuprm_b200.configspace import RobotConfigspace

pytestmark = pytest.mark.gpu


def space(sc):
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND)
    return cs


def launches(cs, call):
    n = cs.stats()["launches"]
    out = call()
    return cs.stats()["launches"] - n, out


SETTINGS = [
    (None, True),
    (lambda cs: cs.set_edge_split(1 << 22), True),          # covers the batch, default segments
    (lambda cs: cs.set_edge_split(40), True),
    (lambda cs: cs.set_edge_split(39), False),              # one warp an edge
    (lambda cs: cs.set_edge_split(0), False),
    (lambda cs: cs.set_edge_split(16384, 1), False),        # segments of the caller's length
    (lambda cs: cs.set_edge_split(16384, 4), False),
    (lambda cs: cs.set_launch(False, 64, False), False),
    (lambda cs: cs.set_launch(True, 64, False), True),      # the other kind's shape
    (lambda cs: cs.profile_enable(True), False),
]


@pytest.mark.parametrize("setting,small", SETTINGS)
def test_edges(setting, small):
    sc = scenes.make_hull6(3)
    qs, qe = scenes.random_edges(sc, 40, 4, 3.0)
    cs = space(sc)
    if setting:
        setting(cs)
    for policy in (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT):
        cs.set_edge_policy(policy)
        ref = space(sc)
        ref.set_edge_policy(policy)
        n, codes = launches(cs, lambda: cs.check_edges(qs, qe))
        np.testing.assert_array_equal(codes, ref.check_edges(qs, qe))
        assert (n == 1) == small


@pytest.mark.parametrize("setting,small", [(None, True), (lambda cs: cs.set_launch(True, 128, True), False),
                                           (lambda cs: cs.set_launch(False, 128, False), True),
                                           (lambda cs: cs.set_edge_split(0), True),
                                           (lambda cs: cs.profile_enable(True), False)])
def test_configurations(setting, small):
    sc = scenes.make_hull6(3)
    q = scenes.uniform_configs(sc, 500, 4)
    cs = space(sc)
    if setting:
        setting(cs)
    n, codes = launches(cs, lambda: cs.check_configs(q))
    np.testing.assert_array_equal(codes, space(sc).check_configs(q))
    assert (n == 1) == small


def test_a_shape_that_does_not_fit_changes_no_route():
    sc = scenes.make_wall7(4)
    cs = space(sc)
    with pytest.raises(Exception):
        cs.set_launch(True, 512, True)
    assert launches(cs, lambda: cs.check_configs(scenes.uniform_configs(sc, 50, 4)))[0] == 1
