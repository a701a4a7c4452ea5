"""The reverse sweep's two ways to divide give the same gradient.

The equations are homogeneous: with the state, the target and WENO-Z's constants scaled by powers of two, every
operation's result scales exactly, the loss by scale^2 and its gradient by scale.  A density of 2^24 lies outside
the range in which the face adjoints divide by shared reciprocals, one near 1 inside it, so the scaled run takes
the IEEE divisions.  Both sum the same contributions in the order of their atomics: the bound between two runs
that differ in that order is 1e-12 of the largest entry, as for the checkpoint intervals.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 17, 17), (5, 7, 11)])  # a dense, and a ragged grid with few faces
@pytest.mark.parametrize("eps,delta", [(1e-6, 0.0), (1e-6, 1e-6)])
def test_scaled_state(awcm_lib, shape, eps, delta):
    from awcm import gradient as G

    s = awcm_lib.AWCM2D(*shape, 0.0, 10.0, 0.0, 10.0, awcm_lib.BC_PERIODIC)
    s.set_q(G.vortex_bumps(s))
    target = G.target_density(s)
    s.prepare(1e-3)
    q = s.get_q()
    out = []
    for scale in (1.0, 2.0**24):
        s.set_wenoz(eps * scale**2, delta * scale**2)
        s.set_q(q * scale)
        loss, grad, _ = s.adjoint(0.0, 2e-3, 7, target * scale)
        out.append((loss / scale**2, grad / scale))
    (l1, g1), (l2, g2) = out
    assert np.abs(g1).max() > 0
    assert l2 == pytest.approx(l1, rel=1e-13)
    assert np.abs(g2 - g1).max() <= 1e-12 * np.abs(g1).max()
