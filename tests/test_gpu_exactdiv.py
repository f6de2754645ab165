"""The device's short quotients (csrc/exactdiv.cuh) against its division, bit for bit: ordinary numbers, divisors next to
powers of two on both sides, quotients next to the middle of two doubles, both sides of every range limit, zeros, infinities
and NaN."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from pyocean_b200 import build as B

pytestmark = pytest.mark.gpu
NAMES = ("quotient", "quot_rn(recip_newton)", "quot_rn(1 / b)", "div3", "div6")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    import torch
    so = str(tmp_path_factory.mktemp("devdiv") / "devdiv.so")
    subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, "-shared", "-o", so,
                    os.path.join(ROOT, "tests", "devcore", "devdiv.cu"), "-lcudart"], check=True)
    L = ctypes.CDLL(so)
    L.check_quotients.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_void_p]

    def run(a, b):
        a, b = np.broadcast_arrays(np.asarray(a, float), np.asarray(b, float))
        ad, bd = (torch.from_numpy(np.ascontiguousarray(x).ravel()).cuda() for x in (a, b))
        wrong = torch.zeros(5, dtype=torch.int64, device="cuda")
        ex = torch.zeros(10, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert L.check_quotients(ad.data_ptr(), bd.data_ptr(), ad.numel(), wrong.data_ptr(), ex.data_ptr()) == 0
        ex = [float(x).hex() for x in ex.cpu()]
        assert wrong.cpu().tolist() == [0] * 5, dict(zip(NAMES, zip(wrong.cpu().tolist(), ex[::2], ex[1::2])))

    return run


def _divisors(rng, n):
    """Mantissas in [1, 2): random; k ulps below 2, above 1 and around the limit of near_two, k odd and even."""
    k = np.concatenate([np.arange(1, n // 8), rng.integers(1, 1 << 36, n // 8)])
    ulp = 2.0 ** -52
    limit = 2.0 - 2.0 ** -18
    return np.concatenate([1.0 + rng.random(n), 2.0 - k * ulp, 1.0 + k * ulp, limit + k * ulp, limit - k * ulp, [1.0, 1.5]])


@pytest.mark.parametrize("seed", range(4))
def test_ordinary_numbers(check, seed):
    rng = np.random.default_rng(seed)
    b = _divisors(rng, 1 << 20)
    b = b * 2.0 ** rng.integers(-390, 390, b.size)
    a = np.resize(_divisors(rng, 1 << 20), b.size)
    rng.shuffle(a)
    check(rng.choice([-1.0, 1.0], b.size) * a * 2.0 ** rng.integers(-480, 480, b.size), b)
    check(a, np.resize(_divisors(rng, 1 << 20), a.size))


def _next_to_midpoints(divisors):
    """53-bit integers A for each odd 53-bit B with A / B next to the middle of two doubles: A 2^e = N B + k, N odd of 54 bits
    (e = 53 for A > B, 54 for A < B), k small."""
    a, b = [], []
    for B in divisors:
        for e in (53, 54):
            inv = pow(1 << e, -1, B)
            for k in (1, 2, 3, 5, 9, -1, -2, -3, -5, -9):
                A = k * inv % B
                A += B if e == 53 else 0
                N = ((A << e) - k) // B
                if 1 << 52 <= A < 1 << 53 and 1 << 53 <= N < 1 << 54 and N & 1:
                    a.append(float(A))
                    b.append(float(B))
    return a, b


def test_quotients_next_to_the_middle_of_two_doubles(check):
    rng = np.random.default_rng(5)
    near = [(1 << 53) - k for k in range(1, 20000, 2)]
    limit = [(1 << 53) - (1 << 34) + d for d in range(-9999, 10000, 2)]
    some = [int(x) | 1 for x in rng.integers(1 << 52, 1 << 53, 20000)]
    for divisors in (near, limit, some):
        a, b = _next_to_midpoints(divisors)
        assert len(a) > 20000
        check(a, b)


def test_range_limits_and_special_values(check):
    e = np.array([-1074, -1073, -1023, -1022, -1021, -1001, -1000, -999, -970, -960, -501, -500, -499, -401, -400, -399, -1, 0,
                  1, 399, 400, 401, 499, 500, 501, 999, 1000, 1001, 1022, 1023])
    m = np.array([1.0, 1.0 + 2.0 ** -52, 1.5, 2.0 - 2.0 ** -17, 2.0 - 2.0 ** -19, 2.0 - 2.0 ** -52])
    with np.errstate(over="ignore", under="ignore"):
        v = (m[:, None] * 2.0 ** e.astype(float)).ravel()
    v = np.concatenate([v, [0.0, np.inf, np.nan, 3.0, 6.0, 0.1]])
    v = np.concatenate([v, -v])
    check(v[:, None], v[None, :])
