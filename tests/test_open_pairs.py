"""Vertex checks of configurations that certificates leave many pairs open
for: links past the ones whose ball is tracked (their pairs are never
certified), and NaN joints (no pair is).  Their lists of exact tests
overflow several times: the codes equal the oracle's in the large kernel
(requests are timed per kernel) and where requests of any size take a block
per 32 configurations, and the time stays in proportion."""
import time

import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_MODE_FAST, GPRM_MODE_FP64_BAND
from gpuprm_b200.configspace import RobotConfigspace
from test_scan import make

pytestmark = pytest.mark.gpu
EXACT, FAST = GPRM_MODE_FP64_BAND, GPRM_MODE_FP64_BAND | GPRM_MODE_FAST

SIZES = [
    (7, 3, 6, False, 0),      # 21 moving links, 5 without a slot
    (7, 3, 60, False, 0),     # the same on 1,395 pairs
    (7, 2, 24, True, 1),      # a static pair left open
    (6, 1, 690, False, 0),    # two sweep groups
]


def space(sc, mode, large=False):
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(mode)
    if large:
        cs.profile_enable(True)
    return cs


@pytest.mark.parametrize("mode", [EXACT, FAST])
@pytest.mark.parametrize("size", SIZES)
def test_codes_equal_the_oracle(size, mode):
    sc = make(*size)
    q = scenes.uniform_configs(sc, 400, 7)
    q[::5, 1] = np.nan
    want = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG)[0]
    for large in (True, False):
        got = space(sc, mode, large).check_configs(q)
        if mode == FAST:
            np.testing.assert_array_equal(got != 0, want != 0)
        else:
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("size", [SIZES[3], (7, 2, 350, False, 0)])
def test_lists_that_overflow_in_both_sweep_groups(size):
    """A band of 10 to 40 cm leaves hundreds of pairs a configuration open."""
    sc = make(*size)
    assert sc.num_pairs > 4096
    q = scenes.uniform_configs(sc, 200, 11)
    for band in (0.1, 0.4):
        want, _, inb = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=band)
        for large in (True, False):
            cs = space(sc, EXACT, large)
            cs.set_band(band)
            np.testing.assert_array_equal(cs.check_configs(q), want)
            s = cs.stats()
            assert s["band_rechecks"] == int(inb.sum())
            assert s["pairs_tested"] > 13 * (want == 0).sum()


@pytest.mark.parametrize("mode", [EXACT, FAST])
def test_many_configurations_by_block_equal_the_large_kernel(mode):
    sc = make(*SIZES[0])
    q = scenes.uniform_configs(sc, 70003, 8)          # four parts of a host request
    by_block, large = space(sc, mode), space(sc, mode, True)
    np.testing.assert_array_equal(by_block.check_configs(q), large.check_configs(q))
    a, b = by_block.stats(), large.stats()
    assert a["band_rechecks"] == b["band_rechecks"] and a["vertex_checks"] == b["vertex_checks"]


def seconds(cs, q, res):
    import torch
    best = 1e9
    for _ in range(10):
        torch.cuda.synchronize()
        t = time.perf_counter()
        cs.check_configs_device(q, res)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def test_nan_configurations_cost_no_more_than_others():
    import torch
    sc = make(*SIZES[3])
    cs = space(sc, EXACT)
    n = 50000
    q = torch.tensor(np.ascontiguousarray(scenes.uniform_configs(sc, n, 9).T), device="cuda:0")
    res = torch.empty(n, dtype=torch.int32, device="cuda:0")
    usual = seconds(cs, q, res)
    q[1] = float("nan")
    assert seconds(cs, q, res) < usual                 # 5 times as long with every open pair's certificates evaluated first


def test_links_without_a_slot_cost_in_proportion():
    import torch
    sc = make(*SIZES[0])
    cs = space(sc, FAST)
    n, m = 200000, 32768
    q = torch.tensor(np.ascontiguousarray(scenes.uniform_configs(sc, n, 10).T), device="cuda:0")
    res = torch.empty(n, dtype=torch.int32, device="cuda:0")
    few = seconds(cs, q[:, :m].contiguous(), res[:m])
    assert seconds(cs, q, res) < 2.0 * n / m * few     # 4.4 times in the large kernel


@pytest.mark.parametrize("mode", [EXACT, FAST])
def test_a_batch_with_links_without_a_slot(mode):
    import torch
    from gpuprm_b200.batch import CONFIGS, ProblemBatch, offsets_of
    scs = [scenes.make_box4(2), make(*SIZES[0]), scenes.make_hull6(3), make(*SIZES[1])]
    counts = [700, 900, 0, 40]
    q = [scenes.uniform_configs(s, n, 12 + n) for s, n in zip(scs, counts)]
    spaces = [space(s, mode) for s in scs]
    want = np.concatenate([space(s, mode).check_configs(x) for s, x in zip(scs, q)])
    offs = offsets_of(counts)
    rows = np.zeros((7, int(offs[-1])), np.float32)
    for x, o in zip(q, offs):
        rows[:x.shape[1], o:o + len(x)] = x.T
    t = torch.tensor(rows, device="cuda:0")
    b = ProblemBatch(spaces)
    b.set_layout(CONFIGS, offs)
    for threshold in (-1, 0, 800):
        b.set_solo_threshold(CONFIGS, threshold)
        res = torch.full((int(offs[-1]),), -7, dtype=torch.int32, device="cuda:0")
        s = b.stats()
        b.check_configs_device(t, res)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(res.cpu().numpy(), want)
        e = b.stats()
        assert e["vertex_checks"] - s["vertex_checks"] == len(want)
        assert e["pairs_tested"] > s["pairs_tested"]
    b.capture(CONFIGS, t, None, res)
    res.fill_(-7)
    b.replay(CONFIGS)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(res.cpu().numpy(), want)


def test_a_batch_of_links_without_a_slot_costs_no_more_than_its_problem():
    import torch
    from gpuprm_b200.batch import CONFIGS, ProblemBatch, offsets_of
    sc = make(*SIZES[0])
    n = 200000
    q = torch.tensor(np.ascontiguousarray(scenes.uniform_configs(sc, n, 10).T), device="cuda:0")
    res = torch.empty(n, dtype=torch.int32, device="cuda:0")
    alone = seconds(space(sc, FAST), q, res)
    b = ProblemBatch([space(sc, FAST)])
    b.set_layout(CONFIGS, offsets_of([n]))
    assert seconds(b, q, res) < 1.5 * alone          # 5 times in the shared launch
