"""Vertex checks on short pair lists, whose certificates go a lane per
configuration: the codes equal the oracle's at and around whole chunks of 32
pairs and the longest list that takes them, with settled static pairs, with
lists of exact tests that overflow (wide bands, NaN joints), and a large
request costs less than its share of a small one."""
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
    (1, 1, 1, False, 0),      # one pair
    (2, 1, 16, False, 0),     # 32 pairs
    (3, 1, 11, False, 0),     # 34 pairs
    (2, 1, 128, False, 0),    # 256 pairs: the longest list
    (1, 1, 257, False, 0),    # one more
    (4, 1, 20, True, 1),      # static pairs: settled ones and one left open
    (4, 1, 20, True, 2),      # nothing is free
    (7, 3, 6, False, 0),      # links without a slot
]


def space(sc, mode, large=True):
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(mode)
    if large:
        cs.set_launch(True, 128, False)
    return cs


def test_sizes_are_the_intended_ones():
    n = [make(*s).num_pairs for s in SIZES]
    assert n[:5] == [1, 32, 34, 256, 257] and max(n[5:]) < 270


@pytest.mark.parametrize("mode", [EXACT, FAST])
@pytest.mark.parametrize("size", SIZES)
def test_codes_equal_the_oracle(size, mode):
    sc = make(*size)
    q = scenes.uniform_configs(sc, 333, 7)
    q[::7, -1] = np.nan
    for band in (1e-5, 0.2):                 # 20 cm: most pairs stay open
        want, _, inb = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=band)
        cs = space(sc, mode)
        cs.set_band(band)
        got = cs.check_configs(q)
        if mode == FAST:
            np.testing.assert_array_equal(got != 0, want != 0)
        else:
            np.testing.assert_array_equal(got, want)
            assert cs.stats()["band_rechecks"] == int(inb.sum())


def test_counters_add_up_on_free_configurations():
    sc = make(3, 1, 11, False, 0)
    cs = space(sc, EXACT)
    q = scenes.uniform_configs(sc, 3000, 9)
    q = q[cs.check_configs(q) == 0]
    s = cs.stats()
    cs.check_configs(q)
    e = cs.stats()
    assert (e["pairs_certified"] - s["pairs_certified"]) + (e["pairs_tested"] - s["pairs_tested"]) == \
        len(q) * sc.num_pairs


def seconds(cs, q, res):
    import torch
    best = 1e9
    for _ in range(20):
        torch.cuda.synchronize()
        t = time.perf_counter()
        cs.check_configs_device(q, res)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def test_a_large_request_costs_less_than_its_share():
    import torch
    sc = scenes.make_box4(3)
    n, m = 1000000, 32768
    q = torch.tensor(np.ascontiguousarray(scenes.uniform_configs(sc, n, 10).T), device="cuda:0")
    res = torch.empty(n, dtype=torch.int32, device="cuda:0")
    cs = space(sc, FAST, False)
    few = seconds(cs, q[:, :m].contiguous(), res[:m])     # by blocks
    assert seconds(cs, q, res) < 0.38 * n / m * few       # 0.27; 0.50 with a sweep per configuration
