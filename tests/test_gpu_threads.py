"""Handles and calls of different sizes in threads side by side: a launch may not depend on what another
thread's launch of the same kernel needs (shared memory among it).  The instances are at their end time,
so that a launch is all there is to a call, and thousands of them meet."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(7, 17), (4, 17), (10, 17), (4, 9)]  # 1025, 129, 8193 and 65 points
CALLS = 3000


def side_by_side(bodies):
    errors, gate = [], threading.Barrier(len(bodies))

    def work(body):
        gate.wait()
        try:
            for _ in range(CALLS):
                body()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_batch_launches(awcm_lib):
    import torch

    torch.cuda.set_device(0)
    lines = []
    for geo in SIZES:  # in decreasing and increasing size
        s = awcm_lib.AWCM1D(*geo, 0.0, 1.0)
        s.init_riemann(0.5, (1.0, 0.0, 1.0), (0.125, 0.0, 0.1))
        s.b.set_run(1e-4, 0.5, 1.0, 1.0)
        lines.append(s)
    side_by_side([lambda b=s.b: b.run_all(1) for s in lines])
    for s in lines:
        assert s.b.status(0)[3] == 1 and s.b.status(0)[4] == 0  # done, no step taken


def test_noalloc_launches(awcm_lib):
    import torch

    torch.cuda.set_device(0)
    bodies, outs = [], []
    for levels, nxc in SIZES:
        w = (nxc - 1) * 2 ** (levels - 1) + 7
        q = torch.ones(3 * w, dtype=torch.float64, device="cuda")
        state = torch.from_numpy(np.zeros(5 * w, np.uint8)).cuda()
        out = torch.zeros(16, dtype=torch.float64, device="cuda")
        outs.append((q, state, out))
        bodies.append(lambda a=(levels, nxc, 0.0, 1.0, 1.4, 0, 1e-4, 0.5, 1.0, 1.0, q.data_ptr(), state.data_ptr(),
                                out.data_ptr(), None): awcm_lib._lib.call("awcm1d_step_noalloc", *a))
    side_by_side(bodies)  # all on one stream: the calls share their scratch
    torch.cuda.synchronize()
    for _, _, out in outs:
        assert out[3].item() == 1 and out[4].item() == 0


def test_creation_beside_launches(awcm_lib):
    import torch

    torch.cuda.set_device(0)
    s = awcm_lib.AWCM1D(*SIZES[0], 0.0, 1.0)
    s.init_riemann(0.5, (1.0, 0.0, 1.0), (0.125, 0.0, 0.1))
    s.b.set_run(1e-4, 0.5, 1.0, 1.0)

    def create(n=[0]):
        n[0] += 1
        if n[0] % 50:
            return
        awcm_lib.AWCM2D(3, 9, 9, 0.0, 1.0, 0.0, 1.0, awcm_lib.BC_TRANSMISSIVE).close()
        awcm_lib.AWCM1D(*SIZES[3], 0.0, 1.0).b.close()

    side_by_side([lambda: s.b.run_all(1), create, create, create])
