"""pairs_certified counts the pairs that a certificate has settled: never a
pair that no certificate can settle (a link past those whose ball is
tracked), whether it was tested or left out behind a collision."""
import numpy as np
import pytest

from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FP32
from gpuprm_b200.configspace import RobotConfigspace
from test_scan import make

TRACKED = 16


def scene():
    """21 moving links among obstacles that most configurations collide with."""
    return make(7, 3, 30, False, 0)


def open_pairs(sc):
    moving = np.flatnonzero(sc.sys > 0)
    late = np.isin(np.arange(len(sc.sys)), moving[TRACKED:])
    return int((late[sc.pair_from] | late[sc.pair_to]).sum())


def test_the_scene_has_pairs_without_a_certificate():
    sc = scene()
    assert 100 < open_pairs(sc) < sc.num_pairs


@pytest.mark.gpu
@pytest.mark.parametrize("large", [False, True])
def test_counts(large):
    sc = scene()
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(GPRM_MODE_FP32)
    if large:
        cs.profile_enable(True)
    most, n = sc.num_pairs - open_pairs(sc), 700
    q = scenes.uniform_configs(sc, n, 3)
    codes = cs.check_configs(q)
    assert (codes != 0).mean() > 0.3
    s = cs.stats()
    assert 0.5 * most * n < s["pairs_certified"] <= most * n
    assert s["pairs_certified"] + s["pairs_tested"] <= sc.num_pairs * n
    qs, qe = scenes.random_edges(sc, 200, 4, 1.5)
    for policy in (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT):
        cs.set_edge_policy(policy)
        before = cs.stats()
        codes = cs.check_edges(qs, qe)
        assert (codes != 0).mean() > 0.3
        s = {k: v - before[k] for k, v in cs.stats().items()}
        assert 0 < s["pairs_certified"] <= most * s["edge_steps_executed"]
        assert s["pairs_certified"] + s["pairs_tested"] <= sc.num_pairs * s["edge_steps_executed"]
