"""The in-place block FFT engine's phase code, run on the CPU, against numpy."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fftblock") / "libfftblock.so"
    src = os.path.join(HERE, "native", "fft_block_check.cpp")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", src, "-o", str(out)])
    lib = ctypes.CDLL(str(out))
    lib.fft_block_check.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    return lib


@pytest.mark.parametrize("r", [4, 6, 8, 10, 12, 14, 16])
@pytest.mark.parametrize("zu", [0, 1])
def test_block_engine_matches_numpy(lib, r, zu):
    """Forward against numpy's FFT and the inverse back to the input, as the
    Stockham engine is held to (2e-7 log2 n); with ``zu`` the upper half of
    the input is zero and never read."""
    n = 256 * r
    rng = np.random.default_rng(r + zu)
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    given = x.copy()
    if zu:
        given[n // 2:] = 1e30
        x[n // 2:] = 0
    out, back = np.empty_like(x), np.empty_like(x)
    assert lib.fft_block_check(r, zu, given.ctypes.data, out.ctypes.data, back.ctypes.data) == 0
    tol = 2e-7 * np.log2(n)
    ref = np.fft.fft(x.astype(np.complex128))
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < tol
    assert np.linalg.norm(back / n - x) / np.linalg.norm(x) < 2 * tol


@pytest.mark.parametrize("cols,stride", [(1, 0), (4, 16 * 288 + 4), (4, 6 * 288 + 4)])
def test_block_engine_accesses_are_free_of_bank_conflicts(lib, cols, stride):
    assert lib.fft_block_conflicts(cols, stride) == 1
