"""The kernels' limited half slopes (minmod, moncen, superbee; van Leer's is a device
function, test_gpu_quotient.py) against half of the reference's expression
(fluxlimiters.F90:109-216), bit for bit, over ordinary differences and the
edges: signed zeros, subnormals, powers of two and their neighbours,
infinities and NaN.  The finite values stay below 2^1022: from there on the
reference's product of the sign sum (2) and a doubled difference is infinite
before it is halved, where half_slope stays finite."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "slope_harness.cu")
DEP = os.path.join(HERE, "..", "piernik_b200", "csrc", "pk_device.cuh")
LIB = os.path.join(HERE, "native", "libslope_harness.so")


@pytest.mark.parametrize("lim", range(1, 4), ids=["minmod", "moncen", "superbee"])
def test_half_slope_is_half_the_slope(lim):
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(SRC), os.path.getmtime(DEP)):
        subprocess.check_call(["nvcc", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC,-O2,-ffp-contract=off",
                               "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, SRC])
    f = C.CDLL(LIB).half_slopes
    tiny, sub = np.finfo(float).tiny, np.finfo(float).smallest_subnormal
    edge = [0.0, sub, 3 * sub, tiny, 1.5 * tiny, 1e-200, 0.75, 1.0, np.nextafter(1.0, 2.0), 3.0, 1e200, 2.0**1021, np.inf, np.nan]
    edge = np.array(edge + [-x for x in edge])
    rng = np.random.default_rng(1)
    rand = rng.standard_normal((2, 20000)) * 10.0 ** rng.integers(-3, 3, (2, 20000))
    dl = np.concatenate([np.repeat(edge, edge.size), rand[0], rand[0], rand[0]])
    dr = np.concatenate([np.tile(edge, edge.size), rand[1], rand[0], -rand[0]])
    got, want = np.empty_like(dl), np.empty_like(dl)
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    f(C.c_int(lim), p(dl), p(dr), C.c_longlong(dl.size), p(got), p(want))
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))
