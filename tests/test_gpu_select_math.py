"""The branch-free square roots and quotients of the tree selects (``csrc/select_math.cuh``), called directly, against ``sqrtf``
and ``/``: equal in every bit on the whole range they are used on."""
import ctypes
import os
import subprocess

import pytest

from mcts_numba_cuda_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("select_math") / "select_math_check.so")
    cmd = [build.nvcc_path()] + build.NVCC_FLAGS + ["-I", os.path.join(build.HERE, "csrc"), "-o", path, os.path.join(HERE, "select_math_check.cu")]
    subprocess.run(cmd, check=True, capture_output=True)
    lib = ctypes.CDLL(path)

    def call(name, *args):
        differ, a, b = ctypes.c_ulonglong(), ctypes.c_float(), ctypes.c_float()
        assert getattr(lib, name)(*args, ctypes.byref(differ), ctypes.byref(a), ctypes.byref(b)) == 0
        return differ.value, a.value, b.value
    return call


# up to 2^25 every mantissa comes with either parity of the exponent; beyond, a count is rounded to one of these first
@pytest.mark.parametrize("first,count,stride", [(1, 1 << 25, 1), (1 << 25, 1 << 20, 1999), (0x7FFFFFFF - (1 << 20) + 1, 1 << 20, 1)])
def test_square_roots_of_counts_round_like_sqrtf(check, first, count, stride):
    assert check("check_roots", first, count, stride)[0] == 0


@pytest.mark.parametrize("first,count,numerators", [(1, 4096, 2048), (4097, (1 << 22) + 1 - 4096, 8)])
def test_quotients_by_counts_round_like_division_and_keep_the_sign_of_zero(check, first, count, numerators):
    differ, a, b = check("check_quotients", first, count, numerators)
    assert differ == 0, f"{differ} quotients differ, one of them {a!r} / {b!r}"
