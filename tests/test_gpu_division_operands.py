"""Divisions by shared reciprocals against IEEE divisions on the same operands, on the device, bit for bit:
the quotient and the reciprocal themselves (every leading significand that the reciprocal's seed can see,
all-ones significands, quotients next to a rounding boundary, signed zeros, exponents over the whole range
that the method claims), the range checks at their edges, and the face fluxes, physical fluxes and wave
speeds built on them: wherever the range checks pass, the results are the IEEE ones, states with NaN,
infinities, zeros and negative pressures or densities among them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    import torch

    torch.cuda.init()
    so = str(tmp_path_factory.mktemp("division") / "division.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "c_pp-library_b200", "csrc"),
                    os.path.join(HERE, "division_device.cu"), "-o", so], check=True)
    return ctypes.CDLL(so)


def up(x):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def p(t):
    return ctypes.c_void_p(t.data_ptr())


def same_bits(a, b):
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


def quotients(dev, a, b):
    import torch

    n = len(a)
    out = torch.empty((n, 4, 2), dtype=torch.float64, device="cuda")
    ta, tb = up(a), up(b)
    assert dev.quotients(p(ta), p(tb), ctypes.c_long(n), p(out)) == 0
    o = out.cpu().numpy()
    eq = same_bits(o[..., 0], o[..., 1])
    eq[:, 1] |= a <= 0  # quot_pos: positive dividends
    return eq


def test_every_seed(dev):
    """The seed of a reciprocal depends on the sign, the exponent and the 20 leading significand bits."""
    rng = np.random.default_rng(20261205)
    head = (np.arange(1 << 20, dtype=np.uint64) << np.uint64(32)) | (np.uint64(1023) << np.uint64(52))
    for low in (np.uint64(0), np.uint64(0xFFFFFFFF), rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64)):
        b = (head | low).view(np.float64)
        a = rng.uniform(1, 2, len(b))
        assert quotients(dev, a, b).all()


def test_adversarial_quotients(dev):
    rng = np.random.default_rng(20261206)
    n = 1 << 20
    ea, eb = rng.integers(-640, 711, n), rng.integers(-640, 711, n)
    ok = np.abs(ea - eb) < 900
    b = rng.uniform(1, 2, n)
    kind = rng.integers(0, 6, n)
    b[kind == 0] = 2 - 2.0 ** -52          # all ones
    b[kind == 1] = 1 + 2.0 ** -52 * rng.integers(0, 4, (kind == 1).sum())
    b[kind == 2] = 2 - 2.0 ** -52 * rng.integers(1, 5, (kind == 2).sum())
    q = rng.uniform(1, 2, n)
    # the dividend nearest to b times a rounding boundary (q and half a unit), in extended precision
    a = (b.astype(np.longdouble) * (q.astype(np.longdouble) + np.longdouble(2.0) ** -53)).astype(np.float64)
    a[kind == 3] = rng.uniform(1, 2, (kind == 3).sum())
    a[kind == 4] = b[kind == 4]
    sa, sb = rng.choice([-1.0, 1.0], (2, n))
    a, b = (sa * np.ldexp(a, ea))[ok], (sb * np.ldexp(b, eb))[ok]
    a[::97] = 0.0
    a[1::97] = -0.0
    assert quotients(dev, a, b).all()


@pytest.mark.parametrize("lo,hi", [(-20, 20), (-100, 30), (-100, 60), (-20, 30), (-60, 700), (-100, 90)])
def test_ranges(dev, lo, hi):
    import torch

    e = [0.0, -0.0, np.nan, np.inf, 5e-324, 2.0 ** -1022, np.finfo(float).max]
    for k in (lo, hi):
        v = 2.0 ** k
        e += [v, np.nextafter(v, 0), np.nextafter(v, np.inf), 2 * v, v / 2]
    x = np.array(e + [-v for v in e])
    out = torch.empty(len(x), dtype=torch.int32, device="cuda")
    tx = up(x)
    assert dev.ranges(p(tx), ctypes.c_long(len(x)), lo, hi, p(out)) == 0
    got = out.cpu().numpy()
    inside = (np.abs(x) >= 2.0 ** lo) & (np.abs(x) < 2.0 ** hi)
    assert np.array_equal(got & 1, ~inside)
    assert np.array_equal(got >> 1, ~(inside | (x == 0)))


def states(rng, n, dim):
    """n faces of six cells: smooth and strong jumps, constant ones, scales inside, at and outside the ranges,
    negative pressures and densities, zeros, NaN and infinities."""
    rho2 = rng.choice([0, 0, 0, -19, 19, -20, 20, -25, 25], n).astype(float)
    u2 = rng.choice([0, 0, 0, 4, 10, -30, -60, -99, 14.5], n)
    jump = rng.choice([0.0, 2.0 ** -40, 1e-6, 0.01, 0.5], n)[:, None]

    def cells(base):
        return base[:, None] * (1 + jump * rng.uniform(-1, 1, (n, 6)))

    rho = cells(rng.uniform(0.2, 2, n)) * 2.0 ** rho2[:, None]
    k = 2.0 ** u2[:, None]
    vel = np.stack([cells(rng.uniform(-2, 2, n) * rng.choice([0.0, 1.0, 1.0], n)) * k for _ in range(dim)])
    pr = cells(rng.uniform(0.1, 2, n)) * rho * k * k
    pr[rng.random((n, 6)) < 0.02] *= -1
    rho[rng.random((n, 6)) < 0.002] *= -1
    q = np.stack([rho, *(rho * vel), pr / 0.4 + 0.5 * rho * (vel * vel).sum(0)], axis=-1)
    # the Riemann states of a tube: two constant sides
    side = rng.random(n) < 0.2
    q[side, :3], q[side, 3:] = q[side, :1], q[side, 5:]
    odd = rng.random(q.shape) < 0.001
    q[odd] = rng.choice([0.0, -0.0, np.nan, np.inf, -np.inf, 2.0 ** -20, 2.0 ** 20, 2.0 ** 30, 2.0 ** -100, 5e-324], odd.sum())
    alpha = (np.abs(vel).max(axis=(0, 2)) + np.sqrt(np.abs(pr / rho).max(axis=1))) * rng.choice([1.0, 1.0, 2.0 ** 40, 0.0], n)
    gamma = rng.choice([1.4, 1.4, 5 / 3, 1.1, 2.0 ** 10], n)
    return q, alpha, gamma


def compare(out, bad, nface):
    half = out.shape[1] // 2
    eq = same_bits(out[:, :half], out[:, half:])
    face, point = eq[:, :nface].all(1), eq[:, nface:].all(1)
    assert face[bad[:, 0] == 0].all() and point[bad[:, 1] == 0].all()
    # both sides of the rule are met
    for k in range(2):
        assert 0.2 < (bad[:, k] == 0).mean() < 0.95


@pytest.mark.parametrize("scheme", [0, 1])
def test_states_1d(dev, scheme):
    import torch

    n = 1 << 19
    q, alpha, gamma = (up(x) for x in states(np.random.default_rng([20261205, scheme]), n, 1))
    out = torch.empty((n, 14), dtype=torch.float64, device="cuda")
    bad = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    assert dev.states1(p(q), p(alpha), p(gamma), ctypes.c_long(n), scheme, p(out), p(bad)) == 0
    compare(out.cpu().numpy(), bad.cpu().numpy(), 3)


@pytest.mark.parametrize("y,eps,delta", [(0, 1e-40, 0.0), (1, 1e-40, 0.0), (0, 1e-6, 1e-6), (1, 1e-2, 0.0)])
def test_states_2d(dev, y, eps, delta):
    import torch

    n = 1 << 19
    q, alpha, gamma = (up(x) for x in states(np.random.default_rng([20261205, y, int(delta * 1e6)]), n, 2))
    out = torch.empty((n, 26), dtype=torch.float64, device="cuda")
    bad = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    assert dev.states2(p(q), p(alpha), p(gamma), ctypes.c_long(n), y, ctypes.c_double(eps), ctypes.c_double(delta),
                       p(out), p(bad)) == 0
    compare(out.cpu().numpy(), bad.cpu().numpy(), 4)
