"""The quotients of the channel models and the receptor chain that carry no range check
(physics.cuh: dp_div_y, fp_over; receptor.cuh: rec_div, rec_quot): Markstein's correction of
a * (1 / b).  The claim is the IEEE quotient over the values that reach them, but for the sign
of a zero (-0 over a positive divisor is +0; every use adds it to something else, or takes its
magnitude or exponential).  Restated in C
(IEEE arithmetic with a fused multiply-add, as on the GPU) and compared bit for bit with
a / b on random operands, on quotients beside a rounding midpoint, on divisors whose
significand is all ones, on zeros, infinities and NaNs; and rec_quot as the device runs it,
on every concentration that reaches it."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>

static double dp_div_y(double a, double b, double y) {
    const double q0 = a * y;
    const double q = fma(fma(-q0, b, a), y, q0);
    return q == q ? q : q0;
}
static float fp_over(float a, float c) {
    const float y = 1.0f / c;
    const float q0 = a * y;
    const float q = fmaf(fmaf(-q0, c, a), y, q0);
    return q == q ? q : q0;
}
static double rec_div(double a, double b, double y) {
    const double q0 = a * y;
    return fma(fma(-q0, b, a), y, q0);
}
/* y0: 1 / b to within 2^-20, what the approximate reciprocal leaves */
static double rec_quot(double a, double b, double y0) {
    double y = y0;
    for (int k = 0; k < 2; k++) y = fma(fma(-b, y, 1.0), y, y);
    return rec_div(a, b, y);
}
static int differ_d(double q, double ref) {
    uint64_t x, z;
    memcpy(&x, &q, 8);
    memcpy(&z, &ref, 8);
    return x != z && !(isnan(q) && isnan(ref)) && !(q == 0.0 && ref == 0.0);
}
long check_dp(const double* a, const double* b, long n) {
    long bad = 0;
    for (long k = 0; k < n; k++) bad += differ_d(dp_div_y(a[k], b[k], 1.0 / b[k]), a[k] / b[k]);
    return bad;
}
long check_rec(const double* a, const double* b, long n) {
    long bad = 0;
    for (long k = 0; k < n; k++) bad += differ_d(rec_div(a[k], b[k], 1.0 / b[k]), a[k] / b[k]);
    return bad;
}
/* every step-th float of [lo, hi], either sign */
long check_fp(float c, uint32_t lo, uint32_t hi, uint32_t step) {
    long bad = 0;
    for (uint32_t u = lo; u <= hi; u += step)
        for (int s = 0; s < 2; s++) {
            const uint32_t v = u | (s ? 0x80000000u : 0u);
            float a;
            memcpy(&a, &v, 4);
            const float q = fp_over(a, c), ref = a / c;
            uint32_t x, z;
            memcpy(&x, &q, 4);
            memcpy(&z, &ref, 4);
            bad += x != z && !(isnan(q) && isnan(ref)) && !(q == 0.0f && ref == 0.0f);
        }
    return bad;
}
/* NMDA's inactivation at every step-th concentration, from reciprocals 2^-20 off either way */
long check_quot(uint32_t lo, uint32_t hi, uint32_t step) {
    long bad = 0;
    for (uint32_t u = lo; u <= hi; u += step) {
        float ca;
        memcpy(&ca, &u, 4);
        const double uM = (double)ca * 1e3f, a = 0.8f * uM, b = uM + 1.0f;
        for (int s = -1; s <= 1; s++) bad += differ_d(rec_quot(a, b, (1.0 + s * 0x1p-20) / b), a / b);
    }
    return bad;
}
"""


def _bits(x):
    return int(np.float32(x).view(np.uint32))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gcc = shutil.which("gcc") or shutil.which("cc")
    if gcc is None:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("quot")
    (d / "q.c").write_text(SRC)
    subprocess.run([gcc, "-O2", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC", str(d / "q.c"), "-o",
                    str(d / "q.so"), "-lm"], check=True)
    lib = C.CDLL(str(d / "q.so"))
    for f in ("check_dp", "check_rec"):
        getattr(lib, f).argtypes = [C.c_void_p, C.c_void_p, C.c_long]
        getattr(lib, f).restype = C.c_long
    lib.check_fp.argtypes = [C.c_float] + [C.c_uint32] * 3
    lib.check_quot.argtypes = [C.c_uint32] * 3
    lib.check_fp.restype = lib.check_quot.restype = C.c_long
    return lib


def _count(f, a, b):
    a, b = np.broadcast_arrays(np.asarray(a, np.float64), np.asarray(b, np.float64))
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return f(a.ctypes.data, b.ctypes.data, a.size)


def _hard(rng, b):
    """dividends whose quotients by b lie beside the midpoint of two doubles"""
    m = rng.randint(1 << 52, 1 << 53, b.size, dtype=np.int64).astype(np.float64)
    return np.concatenate([np.nextafter(m * b, s) for s in (-np.inf, np.inf)] +
                          [m * b + 0.5 * b, np.nextafter(m * b + 0.5 * b, np.inf), np.nextafter(m * b + 0.5 * b, -np.inf)])


@pytest.mark.parametrize("name", ["constants", "volumes", "ghk", "ones"])
def test_dp_div_y(lib, name):
    rng = np.random.RandomState(2)
    n = 200000
    if name == "constants":   # 1000, GAS_CONST * CELSIUS_37 and the time constants and slopes folded at compile time
        f = np.float32
        cs = [1000.0, float(f(8.314) * f(310.15)), 1.5, 100.0, 300.0, 2000.0, 5000.0, 15.0, 5.0] + \
             [float(k) + float(f(1e-6)) for k in (7.0, 13.5, 6.0, 10.0)]
        b = np.array(cs)[rng.randint(0, len(cs), n)]
    elif name == "volumes":   # the charge per mole of volumes from 1e-6 to 1e9 um^3
        b = 96485.0 * np.exp(rng.uniform(np.log(1e-6), np.log(1e9), n)) / 1000.0
    elif name == "ghk":       # 1 - exp(-u), 1e-6 <= |u| <= 20
        u = np.exp(rng.uniform(np.log(1e-6), np.log(20.0), n)) * np.where(rng.rand(n) < 0.5, -1, 1)
        b = 1.0 - np.exp(-u)
    else:
        b = (2.0 - 2.0 ** -52) * 2.0 ** rng.randint(-60, 60, n).astype(np.float64)
    a = rng.standard_normal(n) * 10.0 ** rng.uniform(-200, 200, n)
    assert _count(lib.check_dp, a, b) == 0 and _count(lib.check_rec, a, b) == 0
    k = np.tile(b, 5)
    assert _count(lib.check_dp, _hard(rng, b), k) == 0 and _count(lib.check_rec, _hard(rng, b), k) == 0
    for s in (0.0, -0.0, np.inf, -np.inf, np.nan):
        assert _count(lib.check_dp, s, b) == 0


def test_dp_div_y_by_zero_infinity_and_nan(lib):
    for b in (0.0, np.inf, np.nan):
        assert _count(lib.check_dp, [0.0, 1.0, -1.0, 3e-200, -7e200, np.inf, -np.inf, np.nan], b) == 0


@pytest.mark.parametrize("c", [5.0, 5.5, 6.0, float(np.float32(6.0) + np.float32(1e-6)), 6.2, 10.0,
                               float(np.float32(10.0) + np.float32(1e-6)), 30.1, 968.0])
def test_fp_over(lib, c):
    """dividends from 2^-100 (a potential less a constant is zero or a multiple of 2^-40)"""
    assert lib.check_fp(c, _bits(2.0 ** -100), 0x7F7FFFFF, 997) == 0
    assert lib.check_fp(c, _bits(1e-6), _bits(1e3), 13) == 0
    for a in (0.0, np.inf, np.nan):
        assert lib.check_fp(c, _bits(a), _bits(a), 1) == 0


def test_rec_quot_restated(lib):
    assert lib.check_quot(_bits(1e-9), _bits(1e30), 101) == 0


PROBE = r"""
#include <cstdio>
#include "receptor.cuh"
namespace bnc { namespace {
// Every float from `lo` to `hi`: where rec_quot is not the IEEE quotient, and how often its
// reciprocal is not the nearest double.
__global__ void k_probe(uint32_t lo, uint32_t hi, unsigned long long* bad) {
    unsigned long long q = 0, r = 0;
    for (uint64_t u = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= hi; u += (uint64_t)gridDim.x * blockDim.x) {
        const float ca = __uint_as_float((uint32_t)u);
        const double uM = (double)ca * MM_TO_UM, a = 0.8f * uM, b = uM + 1.0f;
        q += __double_as_longlong(rec_quot(a, b)) != __double_as_longlong(a / b);
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        for (int k = 0; k < 2; k++) y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
        r += __double_as_longlong(y) != __double_as_longlong(1.0 / b);
    }
    if (q) atomicAdd(bad, q);
    if (r) atomicAdd(bad + 1, r);
}
} }
extern "C" int probe(uint32_t lo, uint32_t hi, unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
    int rc = cudaMemset(d, 0, 16) != cudaSuccess;
    if (!rc) bnc::k_probe<<<1184, 256>>>(lo, hi, d);
    rc |= cudaGetLastError() != cudaSuccess;
    rc |= cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


@pytest.mark.gpu
def test_rec_quot_on_the_device(tmp_path):
    from bioneuroncore_b200.build import CSRC, GENCODE, NVCC_FLAGS, _nvcc
    (tmp_path / "p.cu").write_text(PROBE)
    subprocess.run([_nvcc()] + GENCODE + NVCC_FLAGS + ["-I" + CSRC, "-shared", "-o", str(tmp_path / "p.so"),
                                                       str(tmp_path / "p.cu")], check=True)
    lib = C.CDLL(str(tmp_path / "p.so"))
    lib.probe.argtypes = [C.c_uint32, C.c_uint32, C.c_void_p]
    out = (C.c_ulonglong * 2)()
    assert lib.probe(_bits(1e-9), _bits(1e30), out) == 0
    print("reciprocals not the nearest double: %d of %d" % (out[1], _bits(1e30) - _bits(1e-9) + 1))
    assert out[0] == 0
