"""The L2 request of a run of elements stays inside the entries that the operator reads
(csrc/l2_run.hpp, checked on the host over the layouts that the entry points accept)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libparanumal_gb300", "csrc")
SRC = """
#include "l2_run.hpp"
extern "C" void run(uint64_t ggeo, int64_t stride, uint64_t wJ, int64_t ws, int Np, int size, int64_t n, int mass,
                    uint64_t* out) {
  const lpg::L2Run r = lpg::l2_factor_run(ggeo, stride, wJ, ws, Np, size, n, mass != 0);
  out[0] = r.lo; out[1] = r.bytes;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("l2")
    src, so = str(d / "run.cpp"), str(d / "run.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, src, "-o", so],
                   check=True)
    f = ctypes.CDLL(so).run
    u, i, c = ctypes.c_uint64, ctypes.c_int64, ctypes.c_int
    f.argtypes = [u, i, u, i, c, c, i, c, ctypes.POINTER(u)]
    return f


def _layouts(Np, size, base):
    """(name, ggeo, stride, wJ, wJ stride), the arrays beginning at `base`"""
    yield "packed", base, 7 * Np, base + 6 * Np * size, 7 * Np
    yield "wJ first", base + Np * size, 7 * Np, base, 7 * Np
    yield "separate", base, 6 * Np, 1 << 40, Np
    yield "separate, padded", base, 6 * Np + Np // 2, 1 << 40, Np
    yield "separate, padded to 7 Np", base, 7 * Np, 1 << 40, 7 * Np
    yield "wJ behind the factors, other stride", base, 6 * Np, base + 6 * Np * size, 6 * Np + 1


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("size", [2, 4, 8])
def test_request_ends_with_the_last_entry_read(lib, N, size):
    Np = (N + 1) ** 3
    out = (ctypes.c_uint64 * 2)()
    for base in (1 << 20, (1 << 20) + size, (1 << 20) + 16 - size):
        for name, g, stride, w, ws in _layouts(Np, size, base):
            for n in (1, 2, 3, 14, 32):
                for mass in (0, 1):
                    lib(g, stride, w, ws, Np, size, n, mass, out)
                    lo, hi = out[0], out[0] + out[1]
                    end = g + ((n - 1) * stride + 6 * Np) * size   # of the last factor read
                    if mass and w == end - (n - 1) * stride * size and (ws == stride or n == 1):
                        end += Np * size   # of wJ behind them
                    assert lo % 16 == 0 and out[1] % 16 == 0
                    assert out[1] == 0 or (g <= lo and hi <= end), (name, n, mass)
                    # and nothing but the units cut at the two ends is left out
                    assert lo - g < 16 and end - hi < 16, (name, n, mass)
