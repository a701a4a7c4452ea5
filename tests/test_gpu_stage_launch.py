"""The 2D stage launches over their whole range, bit for bit against the CPU restatement.

* Euler: one launch takes a stage's x faces, y faces and coarse points from three lists.  Thresholds from "every
  detail is active" to "none is" make the face lists fill the grid, thin out and hold the boundary layers only; grids with
  nx > ny and nx < ny give a y list shorter and longer than the x list.
* Scalar: one launch takes the finest points, which compute their four faces with shared reciprocals where the
  weights' divisors are below 2^700 and with IEEE divisions beyond, and the coarse points.  Fields of 2^0 to
  2^250 lie inside that range, on both sides of it within one field, and outside.
"""
import numpy as np
import pytest

from oracle import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geo", [(5, 11, 5, 0.0, 10.0, 0.0, 4.0), (5, 5, 11, 0.0, 4.0, 0.0, 10.0)])
@pytest.mark.parametrize("tol", [1e-30, 1e-4, 1e-2, 1e30])
def test_euler_lists(awcm_lib, geo, tol):
    g = awcm_lib.AWCM2D(*geo, awcm_lib.BC_PERIODIC)
    o = Oracle2D(*geo, bc_kind=2, kind="port")
    for x in (g, o):
        x.init_problem(2, 2.1, 1.9)
    t = 0.0
    for step in range(5):
        a, b = g.step(tol, 0.3, t, 1e300), o.step(tol, 0.3, t, 1e300)
        assert a[0] == b[0], step
        t += b[0]
        assert np.array_equal(g.get_q()[3:-3, 3:-3], o.get_q()[3:-3, 3:-3]), step
    assert np.array_equal(g.get_masks()[:, 3:-3, 3:-3], o.get_masks()[:, 3:-3, 3:-3])


@pytest.mark.parametrize("log2", [0, 100, 180, 250])
def test_scalar_scales(awcm_lib, log2):
    levels, nxc, scale = 5, 9, 2.0**log2
    n = (nxc - 1) * 2 ** (levels - 1) + 1
    d = 1.0 / n
    geo = (levels, nxc, nxc, 0.5 * d, 1 - 0.5 * d, 0.5 * d, 1 - 0.5 * d)
    x = 0.5 * d + (np.arange(n + 6) - 3) * d
    q = scale * np.exp(-50 * (x[None] - 0.5) ** 2 - 50 * (x[:, None] - 0.4) ** 2)
    o = Oracle2D(*geo, bc_kind=2, kind="port")
    o.set_scalar()
    o.scalar_set_q(q)
    s = awcm_lib.AWCM2DScalar(*geo)
    s.set_q(q)
    t = 0.0
    for step in range(6):
        out = o.scalar_step(1e-4 * scale, 0.4 * d)
        t, m, upd = s.advance(1e-4 * scale, 0.4 * d, t, 1)
        assert m == 1 and upd == out[0], step
        assert np.array_equal(s.get_q()[3:-3, 3:-3], o.scalar_get_q()[3:-3, 3:-3]), step
    assert np.array_equal(s.get_masks(), o.get_masks())
