"""The device's approximate instructions keep the error bounds that cr_math.cuh's
reciprocal, root and cube root sequences start from, and the sequences give the
IEEE operators' bits from them: every high word that the reciprocal and root
seeds read over two binades (and those scaled over the sequences' whole range),
the arguments nearest a midpoint, and every single-precision depth from 2^-30
to 2^30 m."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from dgswem_b200 import build
from test_rounded_ops import RCP_HARD, SEED_ERR, in_range, sqrt_hard

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def found(tmp_path_factory):
    try:
        nvcc = build.nvcc()
    except RuntimeError as e:
        pytest.skip(str(e))
    out = tmp_path_factory.mktemp("rops_gpu") / "rounded_ops_gpu.so"
    # contraction off, as in the strict kernels
    subprocess.run([nvcc, "-ccbin", build.host_cxx(), "-std=c++17", "-O3", "-fmad=false", *build.ARCH, "-shared",
                    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", str(build.CSRC),
                    str(ROOT / "tests" / "native" / "rounded_ops_gpu.cu"), "-o", str(out)], check=True)
    fn = C.CDLL(str(out)).rounded_ops_gpu
    fn.argtypes = [C.POINTER(C.c_double), C.c_int, C.POINTER(C.c_double), C.POINTER(C.c_ulonglong)]
    hard = np.array(RCP_HARD, dtype=np.float64)
    root = np.array(sqrt_hard())
    x = in_range(np.concatenate([hard, hard * 2.0 ** -60, root, root * 2.0 ** -80, 2.0 ** np.arange(-256.0, 256.0)]))
    errs, counts = (C.c_double * 4)(), (C.c_ulonglong * 5)()
    assert fn(x.ctypes.data_as(C.POINTER(C.c_double)), x.size, errs, counts) == 0
    return dict(zip(("rcp", "rsqrt", "log2", "exp2"), errs)), dict(zip(("rcp", "sqrt", "quot", "pow", "left"), counts))


def test_seed_errors(found):
    errs, _ = found
    assert errs["rcp"] <= SEED_ERR
    assert errs["rsqrt"] <= SEED_ERR
    assert errs["log2"] <= 2.0 ** -17  # absolute
    assert errs["exp2"] <= 2.0 ** -19  # of x^(-1/3)


def test_sequences_round_as_the_operators(found):
    _, counts = found
    assert [counts[k] for k in ("rcp", "sqrt", "quot", "pow")] == [0, 0, 0, 0]
    # the rounding test leaves about one depth in 2^17 to the general method
    assert counts["left"] < 60 * 2 ** 23 / 2 ** 16
