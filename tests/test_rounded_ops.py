"""The stage kernel's reciprocal, quotient, square root and cube root
sequences (cr_math.cuh) give the IEEE operators' bits: random arguments, and
every argument whose result lies so near a midpoint between two doubles that
the sequences' analysis does not decide it, with seeds over the whole error
bound of the device's approximate instructions, 2^-19.9 (the largest over
every high word they read)."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
_dp = C.POINTER(C.c_double)
SEED_ERR = 2.0 ** -19.9

# 53-bit X with 2^106 - M X = k for an odd 54-bit M (the divisors of 2^106 - k
# in range), k = 2 and 4; k = 1 is the significand of all ones, k = 3 has none
RCP_HARD = [
    8480179861092514, 8263449212651198, 5276938686109394, 6583997076838894, 5322981989608814, 4619723575576654,
    8716460134775102, 7331062497459854, 7637721365894914, 6628645658878754, 5359079149933474, 7857326865746386,
    5017593869129758, 6260414481236258, 5433304946044738, 5813097674954626, 8340967600624526, 6743444718440206,
    5852518495683566, 8413745725510706, 7302143716234066, 4663060627120798, 6836844636365422, 5527402342438382,
    4797136447748302, 4543885306550786, 8573369051977618, 7440678027627698, 6015585163436338, 7210714368219586,
    6258053705355746, 5059465667261026, 5440503800133692, 7118995707580124, 9002296740580796, 5316991813459108,
    5298352502788820, 7941263984545340, 6004799503160660, 6525673443791140, 8974540322080660, 6629242916101340,
    4764758390727204, 7120733955830052, 7209683550988788, 5384724193248396, 7943203006394820, 4691463364816860,
    8042426583074580, 5778203295494220]


def sqrt_hard(kmax=128):
    """Doubles A 2^s (A of 53 bits, s = 52, 53) with M^2 - 4 A 2^s = k for an
    odd 54-bit M, |k| < kmax: the square roots of k modulo 2^(s+2), by lifting."""
    out = set()
    for s in (52, 53):
        mod = 2 ** (s + 2)
        for k in range(-kmax + 1, kmax):
            if k % 8 != 1:
                continue
            roots = {1, 3, 5, 7}
            for j in range(4, s + 3):
                roots = {y % 2 ** j for x in roots for y in (x, x + 2 ** (j - 2), x + 2 ** (j - 1))
                         if (y * y - k) % 2 ** j == 0}
            for x in roots:
                for m in range(x, 2 ** 54, mod):
                    a, rest = divmod(m * m - k, mod)
                    if m >= 2 ** 53 and rest == 0 and 2 ** 52 <= a < 2 ** 53:
                        out.add(float(a) * 2.0 ** (s - 52))
    return sorted(out)


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("rops") / "rounded_ops_check.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-shared", "-I",
                    str(ROOT / "dgswem_b200" / "csrc"), str(ROOT / "tests" / "native" / "rounded_ops_check.cpp"),
                    "-o", str(out)], check=True)
    L = C.CDLL(str(out))
    L.rounded_rcp.argtypes = L.rounded_sqrt.argtypes = [_dp, C.c_long, C.c_int, C.c_double]
    L.rounded_quot.argtypes = [_dp, _dp, C.c_long]
    L.rounded_pow_third.argtypes = [_dp, C.c_long, C.POINTER(C.c_long)]
    for f in (L.rounded_rcp, L.rounded_sqrt, L.rounded_quot, L.rounded_pow_third):
        f.restype = C.c_long
    return L


def _p(a):
    return np.ascontiguousarray(a, dtype=np.float64), a.size


def _args(n, seed, lo=-256, hi=256):
    rng = np.random.default_rng(seed)
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n)


def in_range(x):
    """Without the significand of all ones, outside the kernels' range test."""
    return x[np.frexp(x)[0] != np.nextafter(1.0, 0.0)]


def test_reciprocal(ops):
    hard = np.array(RCP_HARD, dtype=np.float64)
    x = np.concatenate([hard, hard * 2.0 ** -60, 2.0 ** np.arange(-256.0, 256.0), _args(200_000, 1)])
    x = in_range(x)
    assert ops.rounded_rcp(x.ctypes.data_as(_dp), x.size, 33, SEED_ERR) == 0


def test_square_root(ops):
    hard = np.array(sqrt_hard())
    assert hard.size > 20
    x = np.concatenate([hard, hard * 2.0 ** -80, 2.0 ** np.arange(-256.0, 256.0), _args(200_000, 2),
                        np.nextafter(np.arange(1.0, 2000.0) ** 2, 0.0), np.arange(1.0, 2000.0) ** 2])
    x = in_range(x)
    assert ops.rounded_sqrt(x.ctypes.data_as(_dp), x.size, 33, SEED_ERR) == 0


def test_quotient(ops):
    a, b = _args(2_000_000, 3, -40, 10), _args(2_000_000, 4, -30, 30)
    b[:len(RCP_HARD)] = RCP_HARD
    assert ops.rounded_quot(a.ctypes.data_as(_dp), b.ctypes.data_as(_dp), a.size) == 0


def test_cube_root_near_and_general_agree(ops):
    rng = np.random.default_rng(5)
    x = np.concatenate([10.0 ** rng.uniform(-8, 8, 2_000_000), np.arange(1.0, 1000.0) ** 3,
                        2.0 ** np.arange(-30.0, 31.0), [2.0 ** -31, 2.0 ** 31, 0.0, -1.0]])
    moved = C.c_long()
    assert ops.rounded_pow_third(x[:-1].ctypes.data_as(_dp), x.size - 1, C.byref(moved)) == 0
    assert moved.value < 3000  # exact cubes and powers, out of range, and about one in 2^17
