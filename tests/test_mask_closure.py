"""CheckReconstruction on bit planes, by itself: the step's device code compiled for the CPU (one warp, its
lanes in turn) against the oracle's CheckReconstruction, on masks without the boundary layers that the
step's chain adds before it.  Details at both ends of a row, where a stencil is one-sided and its marks reach
farthest from the detail, and random masks; rows of several to a warp, of one and of several warps a
row, every width up to four warps a row for the level of spacing 16 (its columns are 32 points apart, so
the words that share a row's last details fall on every lane)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import Oracle2D

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def close_plane(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("closure") / "closure.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "c_pp-library_b200", "csrc"), "-isystem", cuda,
                    os.path.join(HERE, "mask_closure_host.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).close_plane
    f.argtypes = [ctypes.c_int] * 5 + [ctypes.c_void_p]
    return f


def check(close_plane, geo, mask, t0=0):
    """mask: the (ny, nx) points; levels finer than 2^t0 must have no details in it."""
    o = Oracle2D(*geo, 0.0, 1.0, 0.0, 1.0, bc_kind=0, kind="port")
    m = np.zeros((5, o.ny + 6, o.nx + 6), np.uint8)
    m[1, 3:-3, 3:-3] = mask
    o.set_masks(m)
    o.manager(1, 0)
    want = o.get_masks()[1, 3:-3, 3:-3]
    nwx = (o.nx + 6 + 31) // 32
    bits = np.ones((o.ny + 6, 32 * nwx), np.uint8)  # set off the plane, as the chain has them
    bits[:, :o.nx + 6] = m[1]
    plane = np.packbits(bits, axis=1, bitorder="little")
    assert close_plane(o.nx, o.ny, geo[0] - 1, nwx, t0, plane.ctypes.data) == 0
    got = np.unpackbits(plane, axis=1, bitorder="little")
    assert np.array_equal(got[3:-3, 3:o.nx + 3], want), geo
    assert got[:, o.nx + 6:].all() and not got[:3, :o.nx + 6].any()


@pytest.mark.parametrize("chunk", range(4))
def test_end_details_every_width(close_plane, chunk):
    for k in range(26 + 26 * chunk, 52 + 26 * chunk):
        geo = (6, k + 1, 5)
        nx, ny = 32 * k + 1, 129
        mask = np.zeros((ny, nx), bool)
        # the first and the last details of the level, on rows of each kind, far enough apart to tell
        mask[32, nx - 1 - 16] = mask[112, 16] = True
        check(close_plane, geo, mask, t0=4)


@pytest.mark.parametrize("geo", [(2, 5, 5), (4, 8, 5), (5, 9, 7), (6, 16, 5), (6, 33, 5), (6, 61, 5), (7, 31, 5),
                                 (8, 16, 5), (6, 90, 5)])
def test_every_level(close_plane, geo):
    nx, ny = ((n - 1) * 2 ** (geo[0] - 1) + 1 for n in geo[1:])
    rng = np.random.default_rng([20261205, *geo])
    for density in (0.0, 0.0005, 0.02):
        mask = rng.random((ny, nx)) < density
        for t in range(geo[0] - 1):
            h = 1 << t
            mask[rng.integers(0, ny // h) * h, [h, nx - 1 - h]] = True
        check(close_plane, geo, mask)
