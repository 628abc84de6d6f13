"""The double-float arithmetic of the solver's sums and quotients (vare_gb300/csrc/reduce.cuh), compiled
for the host from that header and checked on the CPU against 64 bits.

df_ratio: alpha and beta of the PCG. Before it, they were FP64 quotients rounded to FP32; an exact
quotient rounded once is off by half an ulp at most. The correction's own error is 2^-24 of a
correction of at most an ulp, so the pair's result is off by 0.5 + 2^-22 ulp at most, over every
exponent that a sum of squares in FP32 can have.

df_add: partial sums of up to kBoraMaxReduceBlocks blocks, added as part_collect does. An addition of
two pairs of one sign is off by 3 * 2^-48 at most (Joldes, Muller and Popescu, ACM TOMS 44, 2017);
19 + 5 + 3 of them follow one another, so the sum is off by 2^-41 at most.

residual_scale: a power of two, so that the V-cycle's scaling of the residual and its undoing round
nothing, with the scaled norm in [1, 2)."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

from vare_gb300 import build

SRC = r"""
#include "reduce.cuh"
extern "C" void ratios( int n, const float* a, const float* b, float* out )
{
    for( int i = 0; i < n; ++i )
        out[i] = df_ratio( make_float2( a[2 * i], a[2 * i + 1] ), make_float2( b[2 * i], b[2 * i + 1] ) );
}
extern "C" void add( int n, const float* a, const float* b, float* out )
{
    for( int i = 0; i < n; ++i )
    {
        const DF s = df_add( DF{ a[2 * i], a[2 * i + 1] }, DF{ b[2 * i], b[2 * i + 1] } );
        out[2 * i] = s.hi;
        out[2 * i + 1] = s.lo;
    }
}
extern "C" void scales( int n, const double* rr, float* out )
{
    for( int i = 0; i < n; ++i ) out[i] = residual_scale( rr[i] );
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair")
    src, so = d / "pair.cu", d / "pair.so"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "-I", os.path.join(build.HERE, "csrc"), str(src), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def _call(f, a, b, width):
    out = np.zeros((len(a), width), np.float32)
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    f(len(a), p(a), p(b), p(out))
    return out


def _pairs(x):
    hi = x.astype(np.float32)
    return np.stack([hi, (x - hi).astype(np.float32)], 1)


@pytest.mark.parametrize("lo,hi", [(-35, -25), (-25, -10), (-10, 10), (10, 37)])
def test_ratio(lib, lo, hi):
    rng = np.random.default_rng(1)
    n = 200000
    a = _pairs(10.0 ** rng.uniform(lo, hi, n))
    b = _pairs(10.0 ** rng.uniform(lo, hi, n))
    want = a.astype(np.float64).sum(1) / b.astype(np.float64).sum(1)
    keep = (want > 1e-30) & (want < 1e30)
    got = _call(lib.ratios, a, b, 1)[:, 0].astype(np.float64)
    ulp = 2.0 ** (np.floor(np.log2(want)) - 23)
    assert (np.abs(got - want) / ulp)[keep].max() <= 0.5 + 2.0 ** -22


@pytest.mark.parametrize("n", [1, 33, 608, 2432])
@pytest.mark.parametrize("spread", [0.1, 6.0])
def test_partial_sums(lib, n, spread):
    rng = np.random.default_rng(n)
    x = 10.0 ** rng.uniform(-spread, spread, n)
    p = _pairs(x)
    threads = 128
    acc = np.zeros((threads, 2), np.float32)
    for base in range(0, n, threads):  # a thread's partial sums in order, then the warps' trees, then the warps
        q = np.zeros((threads, 2), np.float32)
        q[:len(p[base:base + threads])] = p[base:base + threads]
        acc = _call(lib.add, acc, q, 2)
    for o in (16, 8, 4, 2, 1):
        acc = _call(lib.add, acc, np.ascontiguousarray(acc[np.arange(threads) ^ o]), 2)
    t = acc[:1]
    for w in range(1, threads // 32):
        t = _call(lib.add, t, acc[32 * w:32 * w + 1], 2)
    want = math.fsum(p.astype(np.float64).ravel())
    assert abs(float(t.astype(np.float64).sum()) - want) <= 2.0 ** -41 * want


def test_scale(lib):
    rng = np.random.default_rng(2)
    rr = np.concatenate([10.0 ** rng.uniform(-70, 70, 20000), 4.0 ** np.arange(-100, 100), 2.0 * 4.0 ** np.arange(-100, 100)])
    sc = np.zeros(len(rr), np.float32)
    lib.scales(len(rr), rr.ctypes.data_as(ctypes.c_void_p), sc.ctypes.data_as(ctypes.c_void_p))
    assert (np.frexp(sc)[0] == 0.5).all()
    norm = sc.astype(np.float64) * np.sqrt(rr)
    assert norm.min() >= 1.0 and norm.max() < 2.0
    r = rng.standard_normal(len(rr)).astype(np.float32) * np.float32(1e-3) / sc
    np.testing.assert_array_equal(r * sc * (np.float32(1) / sc), r)
    rr = np.array([0.0, np.inf, np.nan, 1e-300, 1e300])
    sc = np.zeros(len(rr), np.float32)
    lib.scales(len(rr), rr.ctypes.data_as(ctypes.c_void_p), sc.ctypes.data_as(ctypes.c_void_p))
    assert (sc[:3] == 1).all() and np.isfinite(sc).all() and (sc > 0).all()
