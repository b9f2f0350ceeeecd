"""The FP64 path's quotient by a shared reciprocal, its half slopes on the
integer ALUs and its folded halves, operand by operand: the bits of a/b, of
0.5*limiter and of 0.5*a + b, over random bit patterns, neighbouring mantissas, the exponents at which the
quotient changes over to a plain division, subnormals, zeros of either sign,
infinities and NaN."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HOOKS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "hooks")
BUILD = os.path.join(HOOKS, "_build")


def _ops(a, b):
    from vac_gb300 import build
    os.makedirs(BUILD, exist_ok=True)
    so = os.path.join(BUILD, "libfp64_ops.so")
    src = os.path.join(HOOKS, "fp64_ops.cu")
    deps = [src, os.path.join(build.CSRC, "physics.cuh")]
    if not os.path.exists(so) or os.path.getmtime(so) < max(map(os.path.getmtime, deps)):
        subprocess.run([build.nvcc(), build.ARCH, "-O3", "-std=c++17", "-fmad=false",
                        "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                        "-o", so, src], check=True)
    f = C.CDLL(so).fp64_ops
    dp = C.POINTER(C.c_double)
    f.argtypes = [dp, dp, dp, C.c_longlong]
    out = np.empty((10, a.size))
    assert f(*(v.ctypes.data_as(dp) for v in (a, b, out)), a.size) == 0
    return out


def _operands(kind):
    rng = np.random.default_rng({"bits": 1, "near": 2, "edges": 3, "special": 4}[kind])
    n = 1 << 20
    mant = lambda: rng.integers(0, 1 << 52, n, dtype=np.uint64)
    sign = lambda: rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    if kind == "bits":
        a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for _ in range(2))
    elif kind == "near":  # equal exponents and close mantissas: ties and quotients near one
        m = mant()
        d = rng.integers(-3, 4, n).astype(np.int64)
        e = rng.integers(1023 - 99, 1023 + 100, n).astype(np.uint64) << np.uint64(52)
        a = (e | m) | sign()
        b = ((e | m).astype(np.int64) + d).astype(np.uint64) | sign()
    elif kind == "edges":  # exponents about 2^-800, 2^-100, 2^100, 2^800 and the format's ends
        ea = rng.choice([0, 1, 2, 222, 223, 224, 1023, 1822, 1823, 1824, 2045, 2046], n)
        eb = rng.choice([0, 1, 2, 922, 923, 924, 1023, 1122, 1123, 1124, 2045, 2046], n)
        a = ea.astype(np.uint64) << np.uint64(52) | mant() | sign()
        b = eb.astype(np.uint64) << np.uint64(52) | mant() | sign()
    else:
        v = np.array([0.0, -0.0, 1.0, -1.0, 1.5, 3.0, 1 / 3, 5e-324, -5e-324, 2.2e-308, 1e-300,
                      1e300, 1.7e308, -1.7e308, 8.9e307, np.inf, -np.inf, np.nan, 2.0**-100,
                      2.0**100, 2.0**101, 2.0**-800, 2.0**800, 2.0**801, 0.7, -0.7])
        a, b = (w.ravel().view(np.uint64) for w in map(np.ascontiguousarray, np.meshgrid(v, v)))
    return np.ascontiguousarray(a).view(np.float64), np.ascontiguousarray(b).view(np.float64)


@pytest.mark.parametrize("kind", ["bits", "near", "edges", "special"])
def test_quotient_and_half_slopes(gpu_lib, kind):
    a, b = _operands(kind)
    out = _ops(a, b)
    for k, what in ((0, "quotient"), (2, "minmod"), (4, "woodward"), (8, "half plus")):
        got, ref = out[k], out[k + 1]
        bad = ~((got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref)))
        assert not bad.any(), (what, a[bad][:3], b[bad][:3], got[bad][:3], ref[bad][:3])
    with np.errstate(all="ignore"):
        q = a / b
    fin = np.isfinite(q)
    assert np.array_equal(out[1][fin].view(np.uint64), q[fin].view(np.uint64))
    # the reciprocal that the host forms for the cell widths is the device's
    ok = (b >= 2.0**-100) & (b <= 2.0**100)
    assert np.array_equal(out[6][ok], 1.0 / b[ok])
