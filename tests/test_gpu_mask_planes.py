"""The step's mask and level chain on bit planes against the pass-by-pass byte form (the persistent
PrepareEuler) on the same instance: random mask0, random fields, no flow behind them, so that words of
every pattern, both ends of every stencil and levels that no neighbour decides occur.  Geometries: one
CTA for the whole chain, a launch per pass with and without fine levels of their own, coarse grids
that are not powers of two, grids whose width leaves no or many spare bits in a row's last word.
Masks and levels are compared exactly, and so is the density after the inverse transform."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOS = [(2, 5, 5), (3, 9, 7), (4, 8, 5), (4, 17, 17), (6, 5, 9), (7, 5, 5), (5, 17, 12), (6, 17, 9), (7, 11, 7), (8, 9, 5),
        (3, 16, 40), (5, 42, 37)]


@pytest.mark.parametrize("density", [0.0, 0.002, 0.05, 0.6])
@pytest.mark.parametrize("geo", GEOS)
def test_chain_matches_byte_passes(awcm_lib, geo, density):
    rng = np.random.default_rng([20261205, *geo, int(1000 * density)])
    s = awcm_lib.AWCM2D(*geo, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE)
    h, w = s.ny + 6, s.nx + 6
    q = np.zeros((h, w, 4))
    q[..., 0] = 1 + 0.3 * rng.random((h, w))
    q[..., 1:3] = rng.random((h, w, 2)) - 0.5
    q[..., 3] = 3 + rng.random((h, w))
    masks = np.zeros((5, h, w), np.uint8)
    masks[1] = rng.random((h, w)) < density
    masks[1, :3] = masks[1, -3:] = masks[1, :, :3] = masks[1, :, -3:] = rng.random() < 0.5
    masks[1, 3:-3:1 << (geo[0] - 1), 3:-3:1 << (geo[0] - 1)] |= rng.random() < 0.7
    masks[2:] = rng.random((3, h, w)) < 0.1
    levels = rng.integers(0, geo[0], (4, s.ny, s.nx)).astype(np.int32)
    got = []
    for mode in (0, 1):
        s.set_prepare_mode(mode)
        s.set_q(q)
        s.set_masks(masks)
        s.set_levels(levels)
        out = []
        for _ in range(2):  # the second pass starts from levels of the first
            s.prepare(0.05)
            out += [s.get_masks(), s.get_levels(), s.get_q()]
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
