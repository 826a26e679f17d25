"""Requests that run in one launch with a block per configuration or edge
(k_configs_small, k_edges_small): codes of the exact arithmetic equal the
oracle's at the sizes where the mapping changes (one item, one block's
configurations, several blocks per edge, more items than resident blocks),
both entry points and both policies agree with the large path, and a
rejected edge is still reported."""
import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FAST, GPRM_MODE_FP32,
                              GPRM_MODE_FP64_BAND)
from gpuprm_b200.configspace import GprmError, RobotConfigspace

pytestmark = pytest.mark.gpu


def space(sc, dq, mode, policy=GPRM_EDGES_ALL_STEPS):
    cs = RobotConfigspace(sc, dq=dq)
    cs.init()
    cs.set_mode(mode)
    cs.set_edge_policy(policy)
    return cs


def device(cs, call, *arrays):
    import torch
    t = [torch.tensor(np.ascontiguousarray(a.T), device="cuda:0") for a in arrays]
    res = torch.full((arrays[0].shape[0],), -7, dtype=torch.int32, device="cuda:0")
    call(*t, res)
    torch.cuda.synchronize()
    return res.cpu().numpy()


SCENES = {"box4": lambda: scenes.make_box4(2), "hull6": lambda: scenes.make_hull6(3),
          "wall7": lambda: scenes.make_wall7(4, num_obstacles=96)}


@pytest.mark.parametrize("mode", [GPRM_MODE_FP32, GPRM_MODE_FP64_BAND])
@pytest.mark.parametrize("kind", list(SCENES))
def test_configurations_equal_the_oracle(kind, mode):
    sc = SCENES[kind]()
    cs = space(sc, 0.02, mode)
    q = scenes.uniform_configs(sc, 1300, 5)
    q[7] = np.float32(4.0)                     # outside the joint bounds
    q[8, 0] = np.nan                           # passes the bounds check, as in the reference
    want = O.Oracle(sc).check_configs(q, (O.FP32 if mode == GPRM_MODE_FP32 else O.FP32_BAND) | O.DEVICE_TRIG)[0]
    for n in (1, 2, 31, 593, 1300):            # 593 and more: several configurations a block
        np.testing.assert_array_equal(cs.check_configs(q[:n]), want[:n])
    np.testing.assert_array_equal(device(cs, cs.check_configs_device, q), want)
    assert cs.indicator(q[9]) == want[9] and cs.indicator(q[7]) == 1


@pytest.mark.parametrize("mode", [GPRM_MODE_FP32, GPRM_MODE_FP64_BAND, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST])
@pytest.mark.parametrize("kind", list(SCENES))
def test_edges_equal_the_oracle_and_the_large_path(kind, mode):
    sc = SCENES[kind]()
    dq = 0.02
    qs, qe = scenes.random_edges(sc, 592, 6, 2.0)      # up to 100 steps
    qe[3] = qs[3]                                      # one step: 0/0
    orc = O.Oracle(sc)
    omode = (O.FP32 if mode == GPRM_MODE_FP32 else O.FP32_BAND) | O.DEVICE_TRIG
    want = orc.check_edges(qs, qe, dq, omode)[0]
    for policy in (GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT):
        cs, big = space(sc, dq, mode, policy), space(sc, dq, mode, policy)
        big.profile_enable(True)                       # timed per kernel: the large path
        ref = big.check_edges(qs, qe)
        steps = big.stats()["edge_steps_nominal"]
        got = cs.check_edges(qs, qe)
        np.testing.assert_array_equal(got, ref)
        assert cs.stats()["edge_steps_nominal"] == steps
        for n in (1, 9, 40, 150):                      # 16, 16, 8 and 2 blocks an edge
            np.testing.assert_array_equal(cs.check_edges(qs[:n], qe[:n]), ref[:n])
            np.testing.assert_array_equal(device(cs, cs.check_edges_device, qs[:n], qe[:n]), ref[:n])
        if mode & GPRM_MODE_FAST or policy == GPRM_EDGES_EARLY_EXIT:
            np.testing.assert_array_equal(ref != 0, want != 0)
        else:
            np.testing.assert_array_equal(ref, want)


def test_more_edges_than_resident_blocks_on_a_long_pair_list():
    sc = scenes.make_wall7(5, num_obstacles=300)       # 2421 pairs
    assert sc.num_pairs >= 2048
    qs, qe = scenes.random_edges(sc, 1500, 7, 0.4)
    for mode in (GPRM_MODE_FP64_BAND, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST):
        cs, big = space(sc, 0.01, mode), space(sc, 0.01, mode)
        big.profile_enable(True)
        np.testing.assert_array_equal(cs.check_edges(qs, qe), big.check_edges(qs, qe))


def test_rejected_edge_is_reported_and_the_handle_recovers():
    sc = SCENES["box4"]()
    cs = space(sc, 0.02, GPRM_MODE_FP64_BAND)
    qs, qe = scenes.random_edges(sc, 20, 8, 0.5)
    want = cs.check_edges(qs, qe)
    bad = qe.copy()
    bad[4, 1] = np.inf
    with pytest.raises(GprmError):
        cs.check_edges(qs, bad)
    np.testing.assert_array_equal(cs.check_edges(qs, qe), want)


def test_requests_in_flight_together():
    sc = SCENES["hull6"]()
    cs = space(sc, 0.01, GPRM_MODE_FP64_BAND)
    edges = [scenes.random_edges(sc, n, 9 + n, 0.5) for n in (3, 70, 300)]
    want = [cs.check_edges(*e) for e in edges]
    reqs = []
    for qs, qe in edges:
        n = len(qs)
        res = np.zeros(n, np.int32)
        reqs.append((cs.indicator2_async(np.ascontiguousarray(qs.T).reshape(-1), np.ascontiguousarray(qe.T).reshape(-1),
                                         res, n, n), res))
    for (r, res), w in zip(reversed(reqs), reversed(want)):
        cs.indicator2_async_wait(r)
        np.testing.assert_array_equal(res, w)


@pytest.mark.parametrize("kind,n", [("box4", 300), ("box4", 120000), ("hull6", 2000), ("wall7", 40000)])
def test_large_path_rechecks_by_warp_and_by_thread_equal_the_oracle(kind, n):
    """The large path's FP64 recheck takes a warp per item for few items and
    a thread per item for many (a wide band makes many)."""
    sc = SCENES[kind]()
    q = scenes.uniform_configs(sc, n, 15)
    for band in (1e-5, 2e-2):
        cs = space(sc, 0.02, GPRM_MODE_FP64_BAND)
        cs.set_band(band)
        cs.profile_enable(True)
        got = cs.check_configs(q)
        m = min(n, 3000)
        want, _, inb = O.Oracle(sc).check_configs(q[:m], O.FP32_BAND | O.DEVICE_TRIG, band=band)
        np.testing.assert_array_equal(got[:m], want)
        if m == n:
            assert cs.stats()["band_rechecks"] == int(inb.sum())
        small = space(sc, 0.02, GPRM_MODE_FP64_BAND)
        small.set_band(band)
        np.testing.assert_array_equal(small.check_configs(q[:m]), want)
