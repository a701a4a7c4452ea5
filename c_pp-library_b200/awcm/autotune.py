"""Launch-shape autotuner of the batched 1D step kernel.

The step kernel runs one instance per CTA, with up to 512 threads (128 registers a thread); the CTA
size trades occupancy (CTAs resident per SM, i.e. instances in flight) against per-instance
parallelism.  The tuner times a few RK3 steps of the actual batch for each candidate shape on a
throw-away copy of the batch.  Those opening steps have every instance running; towards the end a few
large ones are left, and there only a wide CTA helps.  So it keeps the widest shape within SLACK of
the fastest (active-point updates per second): for 512 tubes of 257 to
8193 points 256 threads open 3 % faster than 512, and the run to the end takes
5.28 s instead of 2.96 in one launch, 9.89 instead of 6.06 with a launch a step.  Lines of one length are no
exception: 512 tubes of 1025 points open 10 to 12 % faster with 128 threads than with 256 and take 0.37 s
to their end instead of 0.31 to 0.33."""
from __future__ import annotations

import time

CANDIDATES = [(128, 0), (256, 0), (384, 0), (512, 0), (128, 2), (256, 2)]
SLACK = 0.1


def tune(make_copy, t_end: float, tol: float = 1e-4, cfl: float = 0.5, steps: int = 40, candidates=CANDIDATES):
    """make_copy() -> fresh AWCM1DBatch at its initial state.  Returns (chosen (threads, ctas_per_sm),
    {shape: updates/s})."""
    import torch

    rates = {}
    from ._lib import AwcmError

    for shape in candidates:
        b = make_copy()
        try:
            b.set_launch(*shape)
        except AwcmError:  # not a valid shape
            b.close()
            continue
        b.set_run(tol, cfl, 0.0, t_end)
        b.steps(3)  # warm-up (also builds the graph)
        b.sync()
        u0 = b.totals()[0]
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        b.steps(steps)
        b.sync()
        dt = time.perf_counter() - t0
        rates[shape] = (b.totals()[0] - u0) / dt
        b.close()
    fastest = max(rates.values())
    best = max((k for k in rates if rates[k] >= (1 - SLACK) * fastest), key=lambda k: (k[0], rates[k]))
    return best, rates
