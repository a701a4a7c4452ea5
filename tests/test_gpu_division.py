"""The face and speed kernels divide by shared reciprocals while their operands are in a safe range and
with IEEE divisions outside it.  Both are correctly rounded, so runs inside the range, outside it and
across its edges equal the CPU restatement bit for bit: shock tubes (both schemes) and the
four-quadrant problem, scaled by powers of two in density (range edges 2^-20 and 2^20) and in
velocity (energy edge 2^30, momentum edge 2^-100), with states that mix cells on either side."""
import numpy as np
import pytest

from oracle import Oracle1D, Oracle2D

pytestmark = pytest.mark.gpu

SCALES = [(0.0, 0.0), (20.5, 0.0), (25.0, 0.0), (-17.5, 0.0), (-25.0, 0.0), (0.0, 14.5), (0.0, 20.0), (0.0, -49.5),
          (0.0, -110.0)]


@pytest.mark.parametrize("right3", [(0.125, 0.0, 0.1), (0.85, 0.6, 0.8)])
@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("rho2,u2", SCALES)
def test_tube(awcm_lib, scheme, rho2, u2, right3):
    n, s, k = 16 * 2 ** 4 + 1, 2.0 ** rho2, 2.0 ** u2
    geo = (5, 17, 0.5 / n, 1 - 0.5 / n)
    g = awcm_lib.AWCM1D(*geo, scheme=scheme)
    o = Oracle1D(*geo, scheme=scheme, kind="port")
    # a density next to 1 (a divisor with an all-ones significand) beside an ordinary one
    left, right = ((1 - 2.0 ** -53) * s, 0.75 * k, 1.0 * s * k * k), (right3[0] * s, right3[1] * k, right3[2] * s * k * k)
    t = 0.0
    for x in (g, o):
        x.init_riemann(0.5, left, right)
    for step in range(8):
        b = o.step(1e-4 * s, 0.5, t, 1e300)
        try:
            a = g.step(1e-4 * s, 0.5, t, 1e300)
        except awcm_lib.AwcmError as e:
            # the schemes' eps (1e-6, 1e-40) is not scaled with the state: where the smoothness is small
            # against it the scheme is linear and drives the pressure below zero at the strong jump
            assert e.status == 5 and right3[0] < 0.5 and min(rho2, u2) < 0
            return
        assert np.array_equal(a, b), step
        t += b[0]
    assert np.array_equal(g.get_q(), o.get_q())
    assert np.array_equal(g.get_masks(), o.get_masks())


@pytest.mark.parametrize("rho2,u2", SCALES)
def test_quadrants(awcm_lib, rho2, u2):
    s, k = 2.0 ** rho2, 2.0 ** u2
    geo = (4, 9, 7, 0.0, 1.0, 0.0, 0.75)
    g = awcm_lib.AWCM2D(*geo, awcm_lib.BC_TRANSMISSIVE)
    o = Oracle2D(*geo, bc_kind=0, kind="port")
    o.init_problem(0, 0.5, 0.4)
    q = o.get_q() * (s * np.array([1.0, k, k, k * k]))
    t = 0.0
    for x in (g, o):
        x.set_q(q)
    for step in range(4):
        b = o.step(1e-3 * s, 0.4, t, 1e300)
        try:
            a = g.step(1e-3 * s, 0.4, t, 1e300)
        except awcm_lib.AwcmError as e:
            assert e.status == 5 and min(rho2, u2) < 0 and step > 0  # as in test_tube
            return
        assert a[0] == b[0], step
        t += b[0]
    assert np.array_equal(g.get_q()[3:-3, 3:-3], o.get_q()[3:-3, 3:-3])
    assert np.array_equal(g.get_masks()[:, 3:-3, 3:-3], o.get_masks()[:, 3:-3, 3:-3])
