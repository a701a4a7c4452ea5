"""Launch shapes of the 1D step kernel between and beside the usual ones: warps that do not divide a line's words,
a CTA limit, and more threads than the kernel runs, which are run as its largest shape; all give the
oracle's run."""
import numpy as np
import pytest

from oracle import Oracle1D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,ctas", [(96, 0), (160, 1), (384, 0), (448, 3), (640, 0)])
@pytest.mark.parametrize("geo", [(4, 9), (8, 12)])
def test_shape(awcm_lib, geo, threads, ctas):
    g, o = awcm_lib.AWCM1D(*geo, 0.0, 1.0), Oracle1D(*geo, 0.0, 1.0, kind="port")
    for x in (g, o):
        x.init_riemann(0.5, (1.0, 0.0, 1.0), (0.125, 0.0, 0.1))
    g.b.set_launch(threads, ctas)
    assert g.run(1e-4, 0.5, 0.05) == o.run(1e-4, 0.5, 0.05)
    assert np.array_equal(g.get_q(), o.get_q())
    assert np.array_equal(g.get_masks(), o.get_masks()) and np.array_equal(g.get_levels(), o.get_levels())


def test_refused_shapes(awcm_lib):
    g = awcm_lib.AWCM1D(4, 9, 0.0, 1.0)
    for threads in (0, 32, 100, 800, 1056):
        with pytest.raises(awcm_lib.AwcmError):
            g.b.set_launch(threads, 0)
