"""gprm_set_band on an initialised handle: the tables and sweep lists of the
new band are in place for the next call, back and forth, with and without
static pairs, and a change costs no more than a few copies."""
import time

import numpy as np
import pytest

import oracle as O
from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_MODE_FP64_BAND
from gpuprm_b200.configspace import RobotConfigspace
from test_scan import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1, 1, False, 0), (4, 1, 20, True, 1), (6, 1, 690, False, 0)])
def test_codes_follow_the_band(size):
    sc = make(*size)
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND)
    q = scenes.uniform_configs(sc, 200, 9)
    for band in (1e-5, 0.2, 1e-3, 0.2, 1e-5):
        cs.set_band(band)
        want, _, inb = O.Oracle(sc).check_configs(q, O.FP32_BAND | O.DEVICE_TRIG, band=band)
        n = cs.stats()["band_rechecks"]
        np.testing.assert_array_equal(cs.check_configs(q), want)
        assert cs.stats()["band_rechecks"] - n == int(inb.sum())


def test_a_change_takes_a_few_copies():
    sc = scenes.make_hull6(3)
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    best = one = 1e9
    q = scenes.uniform_configs(sc, 1, 9)[0]
    for i in range(50):
        t = time.perf_counter()
        cs.set_band(1e-5 + 1e-8 * i)
        best = min(best, time.perf_counter() - t)
        t = time.perf_counter()
        cs.indicator(q)
        one = min(one, time.perf_counter() - t)
    assert best < 2.0 * one          # 4 times with nine copies and a read-back
