"""Pair lists of more than 65,535 entries, whose indices do not fit the
recorded range of an FP64 recheck: every pair is rechecked, so a check that
only a pair past that index decides inside the band keeps its code."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FP64_BAND
from gpuprm_b200.configspace import RobotConfigspace

BAND = 0.03
FILL = 65600


def make():
    """A small scene, and the same one behind FILL copies of a pair of far
    static obstacles: the codes are those of the small one."""
    rng = np.random.default_rng(11)
    links = [scenes._ellipsoid_link(rng) for _ in range(3)]
    obs = [scenes.hull_polytope(scenes.box_points(0.1, 0.1, 0.1) + np.array([0.0, 0.0, z])) for z in (30.0, -30.0)]
    obs += [scenes._random_hull_obstacle(rng) for _ in range(12)]
    sc = scenes._assemble(3, scenes._arm(3), obs, links, [1, 2, 3], "short", {})
    first = np.zeros(FILL, np.int32)
    order = np.argsort(np.concatenate([first, sc.pair_from]), kind="stable")
    return sc, dataclasses.replace(
        sc, pair_from=np.concatenate([first, sc.pair_from])[order].astype(np.int32),
        pair_to=np.concatenate([first + 1, sc.pair_to])[order].astype(np.int32))


def space(sc, policy=GPRM_EDGES_ALL_STEPS):
    cs = RobotConfigspace(sc, dq=0.05)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND)
    cs.set_band(BAND)
    cs.set_edge_policy(policy)
    return cs


def test_scene_is_the_intended_one():
    sc, long = make()
    assert long.num_pairs == sc.num_pairs + FILL > 65535 and (np.diff(long.pair_from) >= 0).all()
    q = scenes.uniform_configs(sc, 300, 1)
    want, _, inb = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=BAND)
    assert (inb & (want != 0)).sum() > 5              # collisions that the recheck decides
    few, _, _ = O.Oracle(long).check_configs(q[:20], O.FP32_BAND | O.DEVICE_TRIG, band=BAND)
    np.testing.assert_array_equal(few, want[:20])


@pytest.mark.gpu
def test_configurations():
    import torch
    sc, long = make()
    n = 300
    q = scenes.uniform_configs(sc, n, 1)
    want, _, inb = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=BAND)
    cs = space(long)
    np.testing.assert_array_equal(cs.check_configs(q), want)
    assert cs.stats()["band_rechecks"] == int(inb.sum())
    t = torch.tensor(np.ascontiguousarray(q.T), device="cuda:0")
    res = torch.full((n,), -7, dtype=torch.int32, device="cuda:0")
    st = torch.cuda.current_stream().cuda_stream
    assert cs.lib.gprm_indicator_batch_device_noalloc(cs.h, C.c_void_p(t.data_ptr()), C.c_void_p(res.data_ptr()), n, n,
                                                      C.c_void_p(st)) == 0
    np.testing.assert_array_equal(res.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("policy", [GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT])
def test_edges(policy):
    sc, long = make()
    qs, qe = scenes.random_edges(sc, 200, 2, 1.0)
    want, _ = O.Oracle(sc).check_edges(qs, qe, 0.05, O.FP32_BAND | O.DEVICE_TRIG, band=BAND)
    got = space(long, policy).check_edges(qs, qe)
    if policy == GPRM_EDGES_ALL_STEPS:
        np.testing.assert_array_equal(got, want)
    else:
        np.testing.assert_array_equal(got != 0, want != 0)


@pytest.mark.gpu
def test_batch():
    import torch
    from gpuprm_b200.batch import CONFIGS, ProblemBatch, offsets_of
    sc, long = make()
    q = scenes.uniform_configs(sc, 300, 1)
    want, _, _ = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=BAND)
    b = ProblemBatch([space(sc), space(long)])
    b.set_layout(CONFIGS, offsets_of([300, 300]))
    t = np.zeros((7, 600), np.float32)
    t[:3] = np.concatenate([q, q]).T
    res = torch.full((600,), -7, dtype=torch.int32, device="cuda:0")
    b.check_configs_device(torch.tensor(t, device="cuda:0"), res)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(res.cpu().numpy(), np.concatenate([want, want]))
