"""The manager's ComputeLevel pass of the 2D path between steps' mask chains, which rewrite only the levels that
may differ from 0: after a pass on any level set the next PrepareEuler leaves the oracle's levels."""
import numpy as np
import pytest

import oracle
from oracle import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geo", [(3, 9, 7), (5, 17, 12), (4, 40, 33)])
def test_levels_after_a_pass(awcm_lib, geo):
    rng = np.random.default_rng([20261205, *geo])
    g = awcm_lib.AWCM2D(*geo, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE)
    o = Oracle2D(*geo, 0.0, 1.0, 0.0, 1.0, bc_kind=0, kind="port")
    o.init_problem(0, 0.5, 0.4)
    q = o.get_q()
    q[..., 0] *= 1 + 1e-2 * rng.random(q.shape[:2])
    for x in (g, o):
        x.set_q(q)
        x.prepare(1e-3)
    for level_id in range(4):
        masks = o.get_masks()
        masks[2] = rng.random(masks[2].shape) < 0.3
        for x in (g, o):
            x.set_masks(masks)
            x.manager(oracle.CL, 1, level_id)
        assert np.array_equal(g.get_levels(), o.get_levels())
        for x in (g, o):
            x.set_q(q)
            x.prepare(1e-3)
        assert np.array_equal(g.get_levels(), o.get_levels())
        assert np.array_equal(g.get_masks()[:, 3:-3, 3:-3], o.get_masks()[:, 3:-3, 3:-3])
