"""The kernels of large requests (one warp per 32 configurations, one warp or
one segment per edge) on long pair lists, where requests of a test's size
would take the small-request kernels: the 7-DOF wall's 4,117 pairs, in two
sweep groups, and more or fewer slots than the swept direction test covers,
against the oracle, bit for bit in the exact arithmetic."""
import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FAST, GPRM_MODE_FP64_BAND)
from gpuprm_b200.configspace import RobotConfigspace
from test_scan import make

pytestmark = pytest.mark.gpu

SCENES = {"wall7": lambda: scenes.make_wall7(6), "14 slots": lambda: make(7, 2, 24, True, 1),
          "links without a slot": lambda: make(7, 3, 6, False, 0)}


@pytest.mark.parametrize("mode", [GPRM_MODE_FP64_BAND, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST])
@pytest.mark.parametrize("kind", list(SCENES))
def test_codes_equal_the_oracle(kind, mode):
    sc = SCENES[kind]()
    orc = O.Oracle(sc)
    omode = O.FP32_BAND | O.DEVICE_TRIG
    q = scenes.uniform_configs(sc, 500, 5)
    qs, qe = scenes.random_edges(sc, 60, 6, 2.0)
    want_v, want_e = orc.check_configs(q, omode)[0], orc.check_edges(qs, qe, 0.02, omode)[0]
    assert (want_v == 0).any() and (want_v != 0).any() and (want_e == 0).any() and (want_e != 0).any()
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(mode)

    def same(got, want, exact):
        if exact and not mode & GPRM_MODE_FAST:
            np.testing.assert_array_equal(got, want)
        else:
            np.testing.assert_array_equal(got != 0, want != 0)
    cs.set_launch(True, 128, False)
    n = cs.stats()["launches"]
    same(cs.check_configs(q), want_v, True)
    assert cs.stats()["launches"] > n + 1
    for policy in (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT):
        cs.set_edge_policy(policy)
        for split in ((0, 2), (16384, 1), (16384, 3)):
            cs.set_edge_split(*split)
            n = cs.stats()["launches"]
            same(cs.check_edges(qs, qe), want_e, policy == GPRM_EDGES_ALL_STEPS)
            assert cs.stats()["launches"] > n + 1
