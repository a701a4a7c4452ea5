"""The 1D manager's and transforms' single passes one by one against the oracle, on lines from the smallest
to ones whose masks and levels are converted by launches of their own: random masks and fields, every mask
as the target, all masks, levels and fields compared after each pass.  And their cost: a pass must not
pay for the masks and levels that it does not touch, so it takes a fraction of PrepareEuler, which runs
some twenty of them (the inverse transform aside, which visits every point of the line)."""
import time

import numpy as np
import pytest

import oracle
from oracle import Oracle1D

pytestmark = pytest.mark.gpu

SIZES = [(2, 6), (4, 9), (7, 17), (3, 513), (8, 17), (6, 67), (9, 17), (10, 17), (11, 24), (12, 17), (3, 12000)]


@pytest.mark.parametrize("geo", SIZES)
def test_passes_match_oracle(awcm_lib, geo):
    rng = np.random.default_rng([20261205, *geo])
    g, o = awcm_lib.AWCM1D(*geo, 0.0, 1.0), Oracle1D(*geo, 0.0, 1.0, kind="port")

    def same(what):
        assert np.array_equal(g.get_q(), o.get_q()), what
        assert np.array_equal(g.get_masks(), o.get_masks()), what
        assert np.array_equal(g.get_levels(), o.get_levels()), what

    def field():
        q = np.stack([1 + 0.2 * rng.random(g.nx + 6), rng.random(g.nx + 6) - 0.5, 3 + rng.random(g.nx + 6)], 1)
        for x in (g, o):
            x.set_q(q)

    for density in (0.003, 0.3):
        masks = (rng.random((5, g.nx + 6)) < density).astype(np.uint8)
        field()
        for x in (g, o):
            x.set_masks(masks)
        for k in range(4):
            for op, mask_id, level_id in [(oracle.BAND, k, 0), (oracle.CR, k, 0), (oracle.CL, k, k), (oracle.AAZ, k, 0),
                                          (oracle.CL, k, 3 - k), (oracle.APD, k, 3 - k), (oracle.CR, k, 0)]:
                for x in (g, o):
                    x.manager(op, mask_id, level_id)
                same((op, mask_id))
        for what in ("fwt", "iwt", "interpolate", "apply_bc", "prepare"):
            for x in (g, o):
                f = getattr(x, what)
                f(1e-2) if what in ("fwt", "prepare") else f(2) if what == "iwt" else f(1, 2) if what == "interpolate" else f()
            same(what)
        for x in (g, o):
            x.manager(oracle.RR, 4, 0)
        same("residue")


def test_a_pass_is_a_fraction_of_prepare(awcm_lib):
    def best(call):
        b = awcm_lib.AWCM1D(14, 17, 0.0, 1.0)  # 131073 points
        b.init_riemann(0.5, (1.0, 0.0, 1.0), (0.125, 0.0, 0.1))
        b.prepare(1e-4)
        ts = []
        for _ in range(20):
            t = time.perf_counter()
            call(b)
            ts.append(time.perf_counter() - t)
        b.b.close()
        return min(ts)

    whole = best(lambda b: b.prepare(1e-4))
    passes = {op: best(lambda b, op=op: b.manager(op, 1, 0)) for op in range(6)}
    passes |= {"fwt": best(lambda b: b.fwt(1e-4)), "interpolate": best(lambda b: b.interpolate(4, 3)),
               "apply_bc": best(lambda b: b.apply_bc())}
    assert max(passes.values()) < 0.3 * whole, (passes, whole)
