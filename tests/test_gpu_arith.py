"""The written-out square root and quotient of csrc/arith.cuh against IEEE results
(NumPy's float32 square root and float64 division round correctly, as CUDA's sqrtf
and division do).

sqrt2: every power of two with random significands, all subnormal exponents, zero,
the ends of the range, infinity and NaN. At most one unit in the last place off
anywhere; and, as its error before the last rounding is about 2^-44 of the result,
wrongly rounded in about 2^-44 / 2^-25 x 2 = 4 of 10^6 cases: 2 of 10^5 are allowed.

div_by: equal to the division for quotients and operands away from underflow."""

import ctypes as C
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    so = tmp_path_factory.mktemp("arith") / "arith_check.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    r = subprocess.run([nvcc, "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                        "arch=compute_100a,code=sm_100a", f"-I{ROOT / 'fastprox_b200' / 'csrc'}",
                        str(ROOT / "tests" / "cuda" / "arith_check.cu"), "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(str(so))


def _ptr(a):
    return C.c_void_p(a.ctypes.data)


@pytest.mark.gpu
def test_sqrt_of_pairs(lib):
    rng = np.random.default_rng(0)
    bits = (np.arange(255, dtype=np.uint32)[:, None] << 23) | rng.integers(0, 1 << 23, (255, 1 << 14), dtype=np.uint32)
    sub = np.concatenate([(1 << k) + rng.integers(0, 1 << k, 64) for k in range(23)]).astype(np.uint32)
    edge = np.array([0, 1, 0x7fffff, 0x800000, 0x7f7fffff, 0x7f800000], np.uint32)
    edge = np.concatenate([edge, np.arange(255, dtype=np.uint32) << 23, (np.arange(255, dtype=np.uint32) << 23) + 1])
    x = np.concatenate([bits.ravel(), sub, edge, [0, 0, 0x7fc00000, 0x7fc00000]]).astype(np.uint32).view(np.float32)
    x = np.concatenate([x, rng.permutation(x)])  # halves of a pair far apart, too
    x = np.ascontiguousarray(x[: len(x) // 2 * 2])
    got = np.empty_like(x)
    assert lib.check_sqrt2(_ptr(x), _ptr(got), C.c_long(len(x))) == 0
    want = np.sqrt(x)
    nan = np.isnan(x)
    assert np.isnan(got[nan]).all()
    g, w = got[~nan].view(np.int32).astype(np.int64), want[~nan].view(np.int32).astype(np.int64)
    off = np.abs(g - w)
    worst = x[~nan][off.argmax()]
    assert off.max() <= 1, (off.max(), worst, (off > 1).sum())
    assert (off > 0).mean() <= 2e-5, (off > 0).mean()
    assert (got[x == 0] == 0).all() and np.isinf(got[np.isinf(x)]).all()


@pytest.mark.gpu
def test_quotient_by_reciprocal(lib):
    rng = np.random.default_rng(1)
    n = 1 << 22
    y = np.ldexp(1 + rng.random(n), rng.integers(-300, 300, n))
    x = np.ldexp((1 + rng.random(n)) * rng.choice([-1.0, 1.0], n), rng.integers(-300, 300, n))
    # as a gradient's component over its norm, significands of all ones and of one, ties' neighbours, zero
    y[: n // 4] = np.abs(x[: n // 4]) * (1 + rng.random(n // 4))
    ones = np.nextafter(np.ldexp(1.0, rng.integers(-300, 300, 1 << 16)), 0.0)
    y[n // 4: n // 4 + (1 << 16)] = ones
    x[n // 4 + 1000: n // 4 + 1000 + (1 << 16)] = ones[::-1]
    x[n // 2: n // 2 + (1 << 20)] = y[n // 2: n // 2 + (1 << 20)] * rng.integers(1, 1 << 20, 1 << 20)
    x[-1000:] = 0.0
    got = np.empty(n)
    assert lib.check_div_by(_ptr(x), _ptr(y), _ptr(got), C.c_long(n)) == 0
    bad = got != x / y
    assert not bad.any(), (bad.sum(), x[bad][:3], y[bad][:3], got[bad][:3])
