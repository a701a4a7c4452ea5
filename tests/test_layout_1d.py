"""What a 1D instance keeps in shared memory: the host sizes a launch with the bytes that pick_layout names,
and the kernel picks its layout again from those bytes.  Both must come to the same layout, for every
grid and for any share of an SM that a CTA may have."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("layout") / "layout.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "c_pp-library_b200", "csrc"), "-isystem", cuda,
                    os.path.join(HERE, "layout_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def f(nx, maxl, avail, scalar):
        out = (ctypes.c_long * 3)()
        lib.layout(nx, maxl, ctypes.c_long(avail), int(scalar), out)
        return tuple(out)

    return f


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("ctas", [1, 2, 3, 4, 8])
def test_kernel_and_host_agree(layout, ctas, scalar):
    avail = (228 * 1024 // ctas - 1024 - 2304) & ~15
    for levels in range(2, 14):
        for nxc in range(5, 66):
            nx = (nxc - 1) * 2 ** (levels - 1) + 1
            if nx > 70000:
                break
            tier, cap, size = layout(nx, levels - 1, avail, scalar)
            assert size <= avail
            assert layout(nx, levels - 1, size, scalar) == (tier, cap, size), (levels, nxc)
