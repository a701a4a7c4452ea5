"""The allocation-free 1D step (awcm1d_step_noalloc) at sizes where its shared memory is the tightest: the
largest line that it takes, lines whose lists fill what the field leaves of the SM's shared memory, the
first ones that keep less of their field there, and the smallest.  One step each, against the oracle,
bit for bit."""
import numpy as np
import pytest

from oracle import Oracle1D

pytestmark = pytest.mark.gpu

# (levels, coarse points)
SIZES = [(2, 5), (2, 1077), (2, 1078), (4, 269), (4, 288), (8, 17), (8, 33), (6, 241), (10, 16), (10, 17), (12, 5),
         (3, 2049), (2, 4097)]


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("levels,nxc", SIZES)
def test_step_matches_oracle(awcm_lib, levels, nxc, scheme):
    import torch

    torch.cuda.set_device(0)
    nx = (nxc - 1) * 2 ** (levels - 1) + 1
    geo = (levels, nxc, 0.5 / nx, 1 - 0.5 / nx)
    cpu = Oracle1D(*geo, scheme=scheme, kind="port")
    cpu.init_riemann(0.5, (1.0, 0.0, 1.0), (0.125, 0.0, 0.1))
    w = nx + 6
    q = torch.from_numpy(np.ascontiguousarray(cpu.get_q().T)).cuda()
    state = np.zeros(5 * w, np.uint8)
    state[:w] = 0x01
    state[:3] = state[w - 3:w] = 0xE1
    state = torch.from_numpy(state).cuda()
    out = torch.zeros(16, dtype=torch.float64, device="cuda")
    ref = cpu.step(1e-4, 0.5, 0.0, 1.0)
    awcm_lib._lib.call("awcm1d_step_noalloc", *geo, 1.4, scheme, 1e-4, 0.5, 0.0, 1.0, q.data_ptr(), state.data_ptr(),
                       out.data_ptr(), None)
    torch.cuda.synchronize()
    assert out[1].item() == ref[0] and np.array_equal(out[5:9].cpu().numpy(), ref[2:6])
    assert np.array_equal(q.cpu().numpy().T, cpu.get_q())
    mb = state.cpu().numpy()[:w]
    assert np.array_equal(np.stack([(mb >> b) & 1 for b in (4, 0, 1, 2, 3)]), cpu.get_masks())
