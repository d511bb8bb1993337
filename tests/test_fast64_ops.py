"""The branch-free division, reciprocal and square root of the flux functions and the functions built on
them, operation by operation against the plain operators: on the CPU with seeds of the documented form
(20 leading bits in and out, three roundings), on the GPU with its own.  The operands are the ones next to
rounding boundaries, found from the congruences that define them, and the ends of the ranges."""
import ctypes
import math
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import ROOT, assert_bits_equal

SRC = os.path.join(ROOT, "tests", "fast64_ops.cu")
CSRC = os.path.join(ROOT, "cfd_solver_withcuda_b200", "csrc")
DP, IP = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
DIV, DIV_SIGNED, INV, ROOT_OP, DIV_GM1, RCP_SEED, RSQRT_SEED, SLOPE = 0, 1, 2, 3, 4, 5, 6, 10


def _dp(a):
    return a.ctypes.data_as(DP)


class Ops:
    def __init__(self, lib):
        self.lib = lib

    def __call__(self, k, a, b):
        """(branch-free, plain, bad) of operation k on every (a, b)."""
        a, b = (np.ascontiguousarray(x, np.float64) for x in np.broadcast_arrays(a, b))
        f, p, bad = np.empty_like(a), np.empty_like(a), np.empty(a.shape, np.int32)
        assert self.lib.ops_items(k, a.size, _dp(a), _dp(b), _dp(f), _dp(p), bad.ctypes.data_as(IP)) == 0
        return f, p, bad.astype(bool)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ops") / "ops.so")
    # (No -mfma: with it GCC folds the sign into -fma(b, q, -a), which loses the sign of a zero.)
    subprocess.check_call(["g++", "-x", "c++", "-std=c++17", "-O1", "-ffp-contract=off", "-fPIC", "-shared",
                           "-I/usr/local/cuda/include", "-I" + CSRC, SRC, "-o", out])
    return ctypes.CDLL(out)


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    from cfd_solver_withcuda_b200 import build
    out = str(tmp_path_factory.mktemp("ops") / "ops_gpu.so")
    subprocess.check_call([build.nvcc()] + build.ARCH + ["-std=c++17", "-O3", "--fmad=false", "-Xcompiler", "-fPIC",
                                                         "-shared", "-I" + CSRC, SRC, "-o", out])
    return Ops(ctypes.CDLL(out))


@pytest.fixture(params=[0, 1, 2, pytest.param("gpu", marks=pytest.mark.gpu)])
def ops(request):
    """The operations with seeds rounded to nearest, down and up, and on the GPU."""
    if request.param == "gpu":
        return request.getfixturevalue("device")
    lib = request.getfixturevalue("host")
    lib.ops_seed_rounding(request.param)
    return Ops(lib)


def quotients_beside_boundaries(n):
    """(a, b): b = 2^53 - d with the reciprocals next to a rounding boundary, a from the inverse of b modulo
    2^54, so that a / b lies one unit of 2^-105 / b from the middle of two numbers.  All d below 2^16, those
    next to the square roots of j 2^53 below 2^30, and n others."""
    rng = random.Random(1)
    d = list(range(1, 2 ** 16, 2))
    d += [x for j in range(1, 130) for x in range(math.isqrt(j * 2 ** 53) - 150, math.isqrt(j * 2 ** 53) + 150) if x % 2]
    d += [rng.getrandbits(rng.randint(1, 45)) | 1 for _ in range(n)]
    out = []
    for b in (2 ** 53 - x for x in d):
        inv = pow(b, -1, 2 ** 54)
        for s in (1, -1):
            m = (s * inv) % 2 ** 54
            for shift in (53, 54):
                if m >= 2 ** 53 and (b * m - s) % 2 ** shift == 0 and 2 ** 52 <= (b * m - s) >> shift < 2 ** 53:
                    out.append(((b * m - s) >> shift, b))
    return (np.array([x[i] for x in out], np.float64) for i in (0, 1))


def test_seeds(ops):
    """Relative error of the two seeds over every leading mantissa word, in both binades."""
    rng = np.random.default_rng(7)
    hi = np.arange(2 ** 21, dtype=np.int64) + (1023 << 20)
    for lo in (0, 2 ** 32 - 1, rng.integers(0, 2 ** 32, hi.size)):
        b = ((hi << 32) | lo).view(np.float64)
        assert np.abs(ops(RCP_SEED, 0.0, b)[0] * b - 1.0).max() < 2.0 ** -19
        assert np.abs(ops(RSQRT_SEED, 0.0, b)[0] * np.sqrt(b) - 1.0).max() < 2.0 ** -19


def test_quotients_beside_rounding_boundaries(ops):
    a, b = quotients_beside_boundaries(100000)
    for scale in (1.0, -2.0 ** -300):
        f, p, bad = ops(DIV, a * scale, b * 2.0 ** 20)
        assert not bad.any()
        assert_bits_equal(f, p, "quotient")


def test_reciprocals_beside_rounding_boundaries(ops):
    """1 / b for b just below a power of two (1 / b next to the middle of two numbers), all mantissa bits set
    among them, and for random b."""
    rng = random.Random(2)
    d = [1, 3, 5] + [rng.getrandbits(rng.randint(1, 45)) for _ in range(100000)]
    b = np.array([2 ** 53 - x for x in d] + [rng.getrandbits(52) | 2 ** 52 for _ in range(100000)], np.float64)
    f, p, bad = ops(INV, 1.0, b * 2.0 ** -60)
    assert not bad.any()
    assert_bits_equal(f, p, "reciprocal")


def test_roots_beside_rounding_boundaries(ops):
    """sqrt(a) nearest to the middle m of two numbers, m^2 = a + k 2^-106 for small k, in both binades."""
    out = []
    for bits in (54, 55):
        for k in range(-257, 258):
            if k % 8 != 1:
                continue
            x = 1  # x^2 = k modulo 2^bits, one more bit at a time
            for j in range(3, bits):
                if (x * x - k) % 2 ** (j + 1):
                    x += 2 ** (j - 1)
            for m in (x, -x, x + 2 ** (bits - 1), -x + 2 ** (bits - 1)):
                m %= 2 ** bits
                if 2 ** 53 < m < 2 ** 54 and (m * m - k) % 2 ** bits == 0 and 2 ** 52 <= (m * m - k) >> bits < 2 ** 53:
                    out.append(float((m * m - k) >> bits) * 2.0 ** (bits - 106))
    a = np.array(out)
    assert a.size > 64
    for e in (0, 40, -300):
        f, p, bad = ops(ROOT_OP, 0.0, a * 2.0 ** e)
        assert not bad.any()
        assert_bits_equal(f, p, "root")


def test_subnormal_numerators(ops):
    """Numerators around the smallest subnormals, where a / b is rounded once more: the plain operators' bits
    or the flag; zeros of either sign are not flagged."""
    rng = np.random.default_rng(5)
    bits = np.concatenate([np.arange(1, 2000), rng.integers(1, 2 ** 33, 20000), rng.integers(1, 2 ** 52, 20000)])
    a = bits.astype(np.int64).view(np.float64) * np.where(rng.random(bits.size) < 0.5, -1.0, 1.0)
    b = np.exp2(rng.uniform(-30, 30, bits.size))
    for k in (DIV, DIV_GM1):
        f, p, bad = ops(k, a, b)
        assert_bits_equal(np.where(bad, p, f), p, "quotient")
        f, p, bad = ops(k, np.array([0.0, -0.0]), 3.0)
        assert not bad.any()
        assert_bits_equal(f, p, "zero")


def test_signed_zero_quotients(ops):
    """Zero numerators over denominators of either sign: IEEE's zero, not flagged."""
    a = np.array([0.0, -0.0, 0.0, -0.0, 1.5, -1.5, 1.5, -1.5])
    b = np.array([3.0, 3.0, -3.0, -3.0, 0.7, 0.7, -0.7, -0.7])
    f, p, bad = ops(DIV_SIGNED, a, b)
    assert not bad.any()
    assert_bits_equal(f, p, "quotient")


@pytest.mark.parametrize("case", ["rest", "aligned", "shear", "jump"])
def test_hllc_of_uniform_states_is_evaluated_once(host, case):
    """Faces with zero contact speeds or pressure jumps (gas at rest, uniform streams along the face, a
    shear layer) and with jumps: the plain operators' flux without a second evaluation."""
    host.ops_seed_rounding(0)
    rng = np.random.default_rng(3)
    n = 2000
    th = rng.uniform(0, 2 * np.pi, n)
    nrm = np.stack([np.cos(th), np.sin(th), rng.uniform(0.1, 2, n)], 1)
    nrm[:8, :2] = [(1, 0), (-1, 0), (0, 1), (0, -1)] * 2
    q = np.empty((n, 2, 4))
    q[:, :, 0], q[:, :, 3] = 1.0, 1.0 / 1.4
    q[:, :, 1:3] = 0.0
    if case == "aligned":
        q[:, :, 1:3] = 1.5 * np.stack([-nrm[:, 1], nrm[:, 0]], 1)[:, None]
    if case == "shear":
        q[:, 0, 1:3] = np.stack([-nrm[:, 1], nrm[:, 0]], 1)
        q[:, 1, 0] = 2.0
    if case == "jump":
        q[:, 1, 0], q[:, 1, 3] = 0.125, 0.1
    f, p, bad = np.empty((n, 4)), np.empty((n, 4)), np.empty(n, np.int32)
    host.ops_hllc(n, _dp(q), _dp(nrm), _dp(f), _dp(p), bad.ctypes.data_as(IP))
    assert not bad.any()
    assert_bits_equal(f, p, "flux")


@pytest.mark.parametrize("limiter", [1, 2, 4])  # MinMod, Van Leer, van Albada
def test_limited_slopes_of_special_values(ops, limiter):
    """NaN of either sign (a neighbour's gradient after its state has become non-physical), infinities,
    zeros, products that underflow and ordinary differences: the plain operators' slope, or the flag."""
    v = np.array([0.0, 1e-13, 1e-12, 2e-12, 1e-5, 0.3, 1.0, 7.0, 1e-150, 1e-160, 1e-304, 5e-324, 1e160, 1e308, np.inf])
    v = np.concatenate([v, -v, np.array([0x7ff8000000000000, 0x7fffffffffffffff], np.int64).view(np.float64),
                        np.array([0xfff8000000000000, 0xffffffffffffffff], np.uint64).view(np.float64)])
    a, b = (x.ravel() for x in np.meshgrid(v, v))
    f, p, bad = ops(SLOPE + limiter, a, b)
    f = np.where(bad, p, f)
    assert np.array_equal(np.isnan(f), np.isnan(p))
    assert_bits_equal(np.where(np.isnan(p), 0.0, f), np.where(np.isnan(p), 0.0, p), "slope")
    ordinary = (np.abs(a) < 10) & (np.abs(b) < 10) & (np.abs(a * b) > 1e-140)
    assert not bad[ordinary].any()
