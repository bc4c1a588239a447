"""FP32 U(1) and SU(2) chains do not depend on the compiler's contraction: the update's FMAs stand in
the source, so a build with -fmad=false follows the library bit for bit, by either pass."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from klft_b200 import GaugeField
from klft_b200.build import ARCH, CSRC, NVCC, ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def uncontracted(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pinned") / "pinned.so")
    subprocess.run([NVCC] + ARCH + ["-O3", "-std=c++17", "-fmad=false", "--expt-relaxed-constexpr", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cxx", "pinned_pass.cu"), "-o", so], check=True, timeout=300)
    f = C.CDLL(so).pinned_sweeps
    f.argtypes = [C.c_int, C.POINTER(C.c_int), C.POINTER(C.c_float), C.c_double, C.c_double, C.c_int, C.c_int,
                  C.c_ulonglong, C.c_ulonglong, C.c_int]
    return f


def order(L):
    """Device index of each site, x0 fastest: sub * Vh + half-lattice index."""
    s, sub, h, stride = np.arange(int(np.prod(L))), 0, 0, 1
    for d, n in enumerate(L):
        x, s = s % n, s // n
        sub, h, stride = sub + ((x % 2) << d), h + (x // 2) * stride, stride * (n // 2)
    return sub * stride + h


@pytest.mark.parametrize("group", [0, 1])
@pytest.mark.parametrize("nc,L,beta,delta", [(1, [24, 20, 30], 1.2, 0.15), (2, [12, 8, 10, 16], 2.3, 0.3)])
def test_chain_without_contraction(uncontracted, nc, L, beta, delta, group):
    g = GaugeField(L, nc, "mixed", "hot", 5)
    g.set_stream(31, 4)
    nd, V, at = len(L), int(np.prod(L)), order(L)
    u = g.download().reshape(V, nd, nc, nc)
    dev = np.zeros((nd, nc, V), np.complex64)
    for mu in range(nd):
        for j in range(nc):
            dev[mu, j, at] = u[:, mu, 0, j]
    rc = uncontracted(nc, (C.c_int * 4)(*L), dev.ctypes.data_as(C.POINTER(C.c_float)), beta, delta, 10, 30, 31, 4, group)
    assert rc == 0
    g.metropolis(beta, delta, 10, 30)
    want = g.download().reshape(V, nd, nc, nc)[:, :, 0, :]
    np.testing.assert_array_equal(dev[:, :, at].transpose(2, 0, 1), want.astype(np.complex64))
