"""Where the 2D mask chain changes from one launch of one CTA to a launch per pass: on either side of the line steps
equal the oracle's, and the side below it is not the slower one: a step takes longer on a larger grid."""
import numpy as np
import pytest

from oracle import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geo", [(5, 11, 11), (6, 6, 6), (5, 12, 12), (5, 13, 13), (7, 5, 5), (3, 43, 40)])
def test_steps_match_oracle(awcm_lib, geo):
    g = awcm_lib.AWCM2D(*geo, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE)
    o = Oracle2D(*geo, 0.0, 1.0, 0.0, 1.0, bc_kind=0, kind="port")
    t = 0.0
    for x in (g, o):
        x.init_problem(0, 0.5, 0.45)
    for _ in range(3):
        a, b = g.step(1e-3, 0.4, t, 1e9), o.step(1e-3, 0.4, t, 1e9)
        assert a[0] == b[0]
        t += b[0]
    assert np.array_equal(g.get_q()[3:-3, 3:-3], o.get_q()[3:-3, 3:-3])
    assert np.array_equal(g.get_masks()[:, 3:-3, 3:-3], o.get_masks()[:, 3:-3, 3:-3])
    assert np.array_equal(g.get_levels(), o.get_levels())


def test_a_larger_grid_takes_longer(awcm_lib):
    import time

    import torch

    us = []
    for n in (17, 25):  # 257 x 257, 385 x 385
        g = awcm_lib.AWCM2D(5, n, n, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE)
        g.init_problem(awcm_lib.PROBLEM_QUADRANTS, 0.5, 0.5)
        q, m = g.get_q(), g.get_masks()
        best = 1e9
        for _ in range(6):
            g.set_q(q)
            g.set_masks(m)
            g.advance(1e-3, 0.4, 0.0, 1e9, 1)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            g.advance(1e-3, 0.4, 0.0, 1e9, 60)
            best = min(best, time.perf_counter() - t0)
        us.append(best)
        g.close()
    assert us[0] < us[1], us
