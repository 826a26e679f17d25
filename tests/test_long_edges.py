"""Small batches of long edges: blocks that share an edge give the codes of
the large kernels whatever their number, call after call (they leave their
scratch zeroed), and the batches that take them are no slower for it."""
import time

import numpy as np
import pytest

from gpuprm_b200 import scenes
from gpuprm_b200._abi import (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FAST, GPRM_MODE_FP64_BAND)
from gpuprm_b200.configspace import GprmError, RobotConfigspace

pytestmark = pytest.mark.gpu
POLICIES = [GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT]
SCENES = {"box4": lambda: (scenes.make_box4(2), 0.02), "hull6": lambda: (scenes.make_hull6(5), 0.01),
          "wall7": lambda: (scenes.make_wall7(5, num_obstacles=200), 0.01)}


def space(sc, dq, mode, policy, large=False):
    cs = RobotConfigspace(sc, dq=dq)
    cs.init()
    cs.set_mode(mode)
    cs.set_edge_policy(policy)
    if large:
        cs.profile_enable(True)
    return cs


@pytest.mark.parametrize("policy", POLICIES)
@pytest.mark.parametrize("kind", list(SCENES))
def test_blocks_that_share_an_edge_give_the_codes_of_the_large_kernels(kind, policy):
    sc, dq = SCENES[kind]()
    qs, qe = scenes.random_edges(sc, 592, 6, 12.0)
    qe[::3] = qs[::3] + (qe[::3] - qs[::3]) * np.float32(0.02)      # one or two rounds
    qe[5] = qs[5]
    for mode in (GPRM_MODE_FP64_BAND, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST):
        want = space(sc, dq, mode, policy, True).check_edges(qs, qe)
        assert (want != 0).any() and (want == 0).any()
        cs = space(sc, dq, mode, policy)
        for n in (592, 300, 149, 74, 37, 9, 592):       # 2 to 16 blocks an edge
            np.testing.assert_array_equal(cs.check_edges(qs[:n], qe[:n]), want[:n])


@pytest.mark.parametrize("policy", POLICIES)
def test_a_rejected_edge_leaves_the_scratch_zeroed(policy):
    sc, dq = SCENES["box4"]()
    cs = space(sc, dq, GPRM_MODE_FP64_BAND, policy)
    qs, qe = scenes.random_edges(sc, 100, 8, 12.0)
    want = cs.check_edges(qs, qe)
    for at in (0, 99):
        bad = qe.copy()
        bad[at, 1] = np.inf
        with pytest.raises(GprmError):
            cs.check_edges(qs, bad)
        np.testing.assert_array_equal(cs.check_edges(qs, qe), want)


def seconds(cs, args):
    import torch
    best = 1e9
    for _ in range(12):
        torch.cuda.synchronize()
        t = time.perf_counter()
        cs.check_edges_device(*args)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


# one block an edge, whatever its length, took 1.7 and 2.0 times as long as the
# large kernels on hull6
@pytest.mark.parametrize("kind,policy", [("hull6", POLICIES[0]), ("hull6", POLICIES[1]), ("wall7", POLICIES[1])])
def test_small_batches_of_long_edges_are_no_slower_than_the_large_kernels(kind, policy):
    import torch
    total = [0.0, 0.0]
    for seed in range(4):
        sc = scenes.make_hull6(seed) if kind == "hull6" else scenes.make_wall7(seed, num_obstacles=512)
        qs, qe = scenes.random_edges(sc, 300, 11 + seed, 4.0)
        args = [torch.tensor(np.ascontiguousarray(x.T), device="cuda:0") for x in (qs, qe)]
        args.append(torch.empty(300, dtype=torch.int32, device="cuda:0"))
        for i, large in enumerate((False, True)):
            total[i] += seconds(space(sc, 0.01, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST, policy, large), args)
    assert total[0] < 1.3 * total[1]
