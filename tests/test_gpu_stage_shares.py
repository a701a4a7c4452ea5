"""The stage launch's split of its CTAs between coarse points and faces: grids of two and three levels, whose points
are nearly all coarse, step and run frozen like the oracle, and a stage's time follows its points when
they grow."""
import numpy as np
import pytest

from oracle import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geo", [(2, 5, 5), (2, 80, 90), (2, 200, 130), (3, 70, 60)])
def test_mostly_coarse_grids_match_oracle(awcm_lib, geo):
    g = awcm_lib.AWCM2D(*geo, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE)
    o = Oracle2D(*geo, 0.0, 1.0, 0.0, 1.0, bc_kind=0, kind="port")
    t = 0.0
    for x in (g, o):
        x.init_problem(0, 0.5, 0.5)
    for _ in range(3):
        a, b = g.step(1e-3, 0.4, t, 1e9), o.step(1e-3, 0.4, t, 1e9)
        assert a[0] == b[0]
        t += b[0]
    assert np.array_equal(g.get_q()[3:-3, 3:-3], o.get_q()[3:-3, 3:-3])
    dt = 0.25 * b[0]
    for x in (g, o):
        x.prepare(1e-3)
    g.frozen_run(t, dt, 2)
    o.set_freeze(1)
    for k in range(2):
        o.step(0.0, 1.0, t + k * dt, 1e300, dt)
    assert np.array_equal(g.get_q()[3:-3, 3:-3], o.get_q()[3:-3, 3:-3])


def test_time_follows_the_points(awcm_lib):
    """2049 x 2049 points on two levels against 1025 x 1025, all coarse but a band: 4 times the coarse points, twice
    the faces."""
    ms = []
    for n in (513, 1025):
        g = awcm_lib.AWCM2D(2, n, n, 0.0, 10.0, 0.0, 10.0, awcm_lib.BC_PERIODIC)
        g.init_problem(awcm_lib.PROBLEM_VORTEX, 5.0, 5.0)
        g.prepare(1e-3)
        q = g.get_q()
        best = 1e9
        for _ in range(6):
            g.set_q(q)
            best = min(best, g.frozen_run(0.0, 1e-4, 30)[1])
        ms.append(best)
        g.close()
    assert ms[1] < 3.0 * ms[0], ms
