"""The certificate scan at the sizes where it can go wrong: pair counts at
and around whole chunks of 32, rows of 32 chunks and sweep groups, robots with a base
link (pairs whose polytopes are both in frame 0), and more slots than the
swept direction test covers.  Codes of the exact arithmetic must equal the
oracle's, bit for bit."""
import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FAST,
                              GPRM_MODE_FP64_BAND)
from gpuprm_b200.configspace import RobotConfigspace


def make(ndof, per_frame, nobs, base, near, seed=3):
    """An arm with `per_frame` links in every moving frame, optionally a base
    link, and nobs obstacles; near: some obstacles beside the base link,
    too close for its certificate but not touching it; touch (near=2): one
    obstacle through it."""
    rng = np.random.default_rng(seed)
    links, sys = [], []
    for f in range(0 if base else 1, ndof + 1):
        for _ in range(1 if f == 0 else per_frame):
            links.append(scenes._ellipsoid_link(rng))
            sys.append(f)
    obs = [scenes._random_hull_obstacle(rng) for _ in range(nobs)]
    if near:
        obs[0] = scenes.hull_polytope(scenes.box_points(0.2, 0.05, 0.05) + np.array([0.05, 0.12, 0.0]))
    if near == 2:
        obs[1] = scenes.hull_polytope(scenes.box_points(0.1, 0.3, 0.02) + np.array([0.1, 0.0, 0.0]))
    return scenes._assemble(ndof, scenes._arm(ndof), obs, links, sys, "scan", {})


SIZES = [
    (1, 1, 1, False, 0),      # one pair
    (2, 1, 16, False, 0),     # 32 pairs: one whole chunk
    (3, 1, 11, False, 0),     # 34 pairs: one chunk and two pairs
    (6, 1, 169, False, 0),    # 1024 pairs: one whole group
    (6, 1, 170, False, 0),    # a group and a few pairs
    (6, 1, 681, False, 0),    # 4096 pairs: one whole sweep group
    (6, 1, 690, False, 0),    # a sweep group and a few pairs
    (4, 1, 20, True, 0),      # base link, every static pair settled
    (4, 1, 20, True, 1),      # base link, one static pair left to the exact test
    (4, 1, 20, True, 2),      # base link through an obstacle: nothing is free
    (7, 2, 24, True, 1),      # 14 slots: no swept direction test
    (7, 3, 6, False, 0),      # 21 moving links: some without a slot
]


def test_sizes_are_the_intended_ones():
    n = [make(*s).num_pairs for s in SIZES]
    assert n[0] == 1 and n[1] == 32 and n[2] == 34 and n[3] == 1024 and n[4] == 1030
    assert n[5] == 4096 and n[6] == 4150


def check(sc, cs, exact, nq=400, ne=60):
    q = scenes.uniform_configs(sc, nq, 7)
    qs, qe = scenes.random_edges(sc, ne, 8, 1.2)
    orc = O.Oracle(sc)
    mode = O.FP32_BAND | O.DEVICE_TRIG
    want_v, want_e = orc.check_configs(q, mode)[0], orc.check_edges(qs, qe, 0.02, mode)[0]
    got_v, got_e = cs.check_configs(q), cs.check_edges(qs, qe)
    if exact:
        np.testing.assert_array_equal(got_v, want_v)
        np.testing.assert_array_equal(got_e, want_e)
    else:
        np.testing.assert_array_equal(got_v != 0, want_v != 0)
        np.testing.assert_array_equal(got_e != 0, want_e != 0)


@pytest.mark.gpu
@pytest.mark.parametrize("size", SIZES)
def test_codes_equal_the_oracle(size):
    sc = make(*size)
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_edge_policy(GPRM_EDGES_ALL_STEPS)
    check(sc, cs, True)
    cs.set_edge_split(0)              # one warp per edge
    check(sc, cs, True)
    cs.set_edge_policy(GPRM_EDGES_EARLY_EXIT)
    check(sc, cs, False)
    cs.set_edge_policy(GPRM_EDGES_ALL_STEPS)
    if size[2] <= 24:
        cs.set_launch(True, 128, True)    # scene tables in shared memory
        cs.set_launch(False, 128, True)
        check(sc, cs, True)
    cs.set_mode(GPRM_MODE_FP64_BAND | GPRM_MODE_FAST)
    check(sc, cs, False)


@pytest.mark.gpu
def test_band_change_settles_the_static_pairs_anew():
    sc = make(4, 1, 20, True, 1)
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND)
    q = scenes.uniform_configs(sc, 300, 9)
    for band in (0.3, 1e-5, 2e-2):
        cs.set_band(band)
        want, _, _ = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=band)
        np.testing.assert_array_equal(cs.check_configs(q), want)
